"""Linear layers of the hybrid family at the sizes where their kernels change, against float64.

Products of the operands are formed exactly or in fp32 and summed in fp32: with K terms an error of a few 2^-24 of Σ |x w| per level of the
sum; 2^-20 Σ |x w| bounds every kernel here.  bfloat16 results add one rounding (2^-9)."""
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu

from jax_llama_b200.ops import seq_kernels as SK  # noqa: E402


def check(got, x, w, act=lambda z: z):
    x, w = x.double(), w.double()
    ref = act(x @ w.T)
    bound = 2.0 ** -20 * (x.abs() @ w.abs().T) + (2.0 ** -8 if got.dtype == torch.bfloat16 else 2.0 ** -22) * ref.abs()
    assert bool(((got.double() - ref).abs() <= bound + 1e-30).all()), ((got.double() - ref).abs() - bound).max()


@pytest.mark.parametrize("M", [4, 5, 7, 8])
@pytest.mark.parametrize("N,K", [(1521, 2048), (1536, 8), (1543, 104), (4100, 264), (2048, 5464), (1600, 8200), (33000, 256),
                                  (1543, 1544), (1536, 1528), (33000, 1600), (1536, 24576), (1536, 24584)])
def test_decode_rows_bfloat16(M, N, K):
    g = torch.Generator().manual_seed(N + K + M)
    x, w = torch.randn(M, K, generator=g).bfloat16().cuda(), torch.randn(N, K, generator=g).bfloat16().cuda()
    check(SK.linear(x, w), x, w)
    check(SK.linear(x, w, act=SK.ACT_RELU, out_f32=False), x, w, torch.relu)


def test_decode_rows_of_chosen_matrices():
    """One matrix per batch by index, some batches without one, several rows per batch."""
    g = torch.Generator().manual_seed(3)
    n, rows, N, K = 6, 6, 520, 1992
    x, w = torch.randn(n * rows, K, generator=g).bfloat16().cuda(), torch.randn(4, N, K, generator=g).bfloat16().cuda()
    index = torch.tensor([2, -1, 0, 3, -1, 2], dtype=torch.int32, device="cuda")
    out = torch.full((n * rows, N), 7.0, device="cuda")
    SK.linear_batched(x, w, out, nbatch=n, rows=rows, x_bs=rows * K, o_bs=rows * N, w_index=index)
    for z, e in enumerate(index.tolist()):
        part = slice(z * rows, (z + 1) * rows)
        if e < 0:
            assert bool((out[part] == 7.0).all())
        else:
            check(out[part], x[part], w[e])


@pytest.mark.parametrize("M,N,K", [(9, 1, 256), (9, 300, 260), (31, 129, 1024), (33, 127, 320), (64, 1000, 2052), (65, 128, 5464), (128, 257, 512), (129, 4100, 256),
                                   (300, 3000, 516), (1000, 640, 2048)])
def test_float32_rows(M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    x, w = torch.randn(M, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda()
    check(SK.linear(x, w), x, w)
    check(SK.linear(x, w, act=SK.ACT_RELU), x, w, torch.relu)
    wide = torch.randn(M, K + 12, generator=g).cuda()       # rows of a wider matrix
    check(SK.linear(wide[:, 4:4 + K], w), wide[:, 4:4 + K], w)


def test_float32_is_as_good_as_fused_multiply_add():
    """Six products of three bfloat16 parts: 2^-22 of a sum of 2048 terms, where one part alone is off by 2^-9."""
    g = torch.Generator().manual_seed(5)
    x, w = torch.randn(100, 2048, generator=g).cuda(), torch.randn(500, 2048, generator=g).cuda()
    ref = x.double() @ w.double().T
    assert float((SK.linear(x, w).double() - ref).norm() / ref.norm()) < 2.0 ** -22


def test_float32_batches_and_sorted_rows():
    g = torch.Generator().manual_seed(6)
    n, rows, N, K = 5, 20, 140, 384
    x, w = torch.randn(n * rows, K, generator=g).cuda(), torch.randn(4, N, K, generator=g).cuda()
    index = torch.tensor([2, -1, 0, 3, 2], dtype=torch.int32, device="cuda")
    out = torch.full((n * rows, N), 7.0, device="cuda")
    SK.linear_batched(x, w, out, nbatch=n, rows=rows, x_bs=rows * K, o_bs=rows * N, w_index=index)
    for z, e in enumerate(index.tolist()):
        part = slice(z * rows, (z + 1) * rows)
        assert bool((out[part] == 7.0).all()) if e < 0 else check(out[part], x[part], w[e]) is None
    group = torch.tensor([1, -1, 3], dtype=torch.int32, device="cuda")              # tiles of 64 sorted rows
    src = torch.randint(0, n * rows, (192,), generator=g).to(torch.int32)
    src[50:64] = -1                                                                 # padding rows read as zero
    out = torch.full((192, N), 7.0, device="cuda")
    SK.linear_sorted(x, w, out, group, src.cuda())
    gathered = torch.where(src[:, None].cuda() >= 0, x[src.clamp_min(0).long().cuda()], torch.zeros((), device="cuda"))
    check(out[:64], gathered[:64], w[1])
    check(out[128:], gathered[128:], w[3])
    assert bool((out[64:128] == 7.0).all()) and bool((out[50:64] == 0.0).all())


def test_float32_infinities_and_nan_stay_what_they_are():
    x, w = torch.ones(20, 512, device="cuda"), torch.randn(300, 512, generator=torch.Generator().manual_seed(7)).cuda()
    x[3, 100], x[5, 7], x[6, 8] = float("inf"), float("nan"), 3.0e38
    w[9, 200] = float("-inf")
    w[10, 8] = 3.0e38
    got, want = SK.linear(x, w), (x.double() @ w.double().T).float()
    same = torch.isfinite(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    assert torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
    keep = same & (torch.arange(20, device="cuda")[:, None] != 6)
    assert float((got - want)[keep].abs().max()) < 1e-3


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (257, 264, 72), (300, 2048, 5464), (511, 520, 128), (600, 1032, 264), (1000, 776, 2048)])
def test_prompt_rows_bfloat16_on_cta_pairs(M, N, K):
    """fp32 and bfloat16 results of ragged sizes (the last tile of rows, columns and K is cut off by the tensor maps): nothing beyond them is
    written.  Sums of K products by a tensor core that cuts off: 2^-17 Σ |x w| is four times what 5464 terms give."""
    g = torch.Generator().manual_seed(M + N)
    x, w = torch.randn(M, K, generator=g).bfloat16().cuda(), torch.randn(N, K, generator=g).bfloat16().cuda()
    room = torch.full((M * N + 4096,), 7.0, device="cuda")
    got = SK.linear(x, w, out=room[:M * N].view(M, N))
    ref, scale = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    assert bool(((got.double() - ref).abs() <= 2.0 ** -17 * scale + 1e-30).all())
    assert bool((room[M * N:] == 7.0).all())
    room = torch.full((M * N + 4096,), 7.0, dtype=torch.bfloat16, device="cuda")
    got = SK.linear(x, w, out_f32=False, out=room[:M * N].view(M, N))
    assert bool(((got.double() - ref).abs() <= 2.0 ** -17 * scale + 2.0 ** -8 * ref.abs() + 1e-30).all())
    assert bool((room[M * N:] == 7.0).all())


@pytest.mark.parametrize("how", ["argument", "environment"])
def test_exact_kernels_are_still_there(how, monkeypatch):
    """`tensor_cores=False` and JLLAMA_HYBRID_TC=0: the SIMT kernels, shown bit for bit by the same rows in calls that no tensor-core kernel
    takes (four rows at a time in bfloat16, rows off the 16-byte boundary in float32).  The tensor-core kernels order their sums in another way."""
    g = torch.Generator().manual_seed(8)
    x, w = torch.randn(8, 2048, generator=g).bfloat16().cuda(), torch.randn(2048, 2048, generator=g).bfloat16().cuda()
    exact = torch.cat([SK.linear(x[:4], w), SK.linear(x[4:], w)])
    xf, wf = torch.randn(100, 2048, generator=g).cuda(), torch.randn(500, 2048, generator=g).cuda()
    odd = torch.empty(100, 2049, device="cuda")
    odd[:, :2048] = xf
    exact_f = SK.linear(odd[:, :2048], wf)
    fast, fast_f = SK.linear(x, w), SK.linear(xf, wf)
    kw = {}
    if how == "argument":
        kw = dict(tensor_cores=False)
    else:
        monkeypatch.setenv("JLLAMA_HYBRID_TC", "0")
        out = torch.empty(8, 2048, device="cuda")
        assert torch.equal(SK.linear_batched(x, w[None], out, nbatch=1, rows=8, x_bs=0, o_bs=0), exact)
        out = torch.empty(100, 500, device="cuda")
        assert torch.equal(SK.linear_batched(xf, wf[None], out, nbatch=1, rows=100, x_bs=0, o_bs=0), exact_f)
    assert torch.equal(SK.linear(x, w, **kw), exact) and torch.equal(SK.linear(xf, wf, **kw), exact_f)
    assert not torch.equal(fast, exact) and not torch.equal(fast_f, exact_f)


@pytest.mark.parametrize("M,N,K", [(20, 64, 256), (100, 500, 2048)])
def test_float32_of_one_sign_is_not_biased(M, N, K):
    """Operands of one sign whose lower parts are as large as they get: products left out would all pull the same way.  Rounded parts leave out
    less than 2^-24 of a product; the tensor core cuts off some thirty times per 64 products, most of it in the last four (2^-23 of the sum
    each at most), and the sums of 64 round once each: 2^-21 holds with room, parts cut off instead of rounded miss it (2^-21 alone)."""
    worst = 1 + 2.0 ** -7 - 2.0 ** -23
    x, w = torch.full((M, K), worst, device="cuda"), torch.full((N, K), worst, device="cuda")
    ref = x.double() @ w.double().T
    assert float(((SK.linear(x, w).double() - ref) / ref).abs().max()) < 2.0 ** -21
    g = torch.Generator().manual_seed(K)
    x, w = torch.rand(M, K, generator=g).cuda(), torch.rand(N, K, generator=g).cuda()
    ref = x.double() @ w.double().T
    assert float(((SK.linear(x, w).double() - ref) / ref).mean().abs()) < 2.0 ** -22


def test_a_short_k_first_does_not_set_the_number_of_resident_pairs():
    """The persistent grid of the CTA-pair kernel is as wide as what fits at its own ring depth, whatever ran before it in the process."""
    code = ("import sys, torch\n"
            "from jax_llama_b200.ops import _lib, seq_kernels as SK\n"
            "for K in map(int, sys.argv[1:]):\n"
            "    SK.linear(torch.zeros(2048, K, dtype=torch.bfloat16, device='cuda'), torch.zeros(2048, K, dtype=torch.bfloat16, device='cuda'))\n"
            "print(_lib.lib().jl_gemm_2cta_pairs())\n")
    last = [subprocess.run([sys.executable, "-c", code, *ks], capture_output=True, text=True, timeout=120, check=True).stdout.split()[-1]
            for ks in (["512"], ["64", "512"])]
    assert last[0] == last[1] and int(last[0]) > 0


@pytest.mark.parametrize("N,K", [(1536, 2048), (2048, 1536), (8192, 2048), (2048, 5464), (2048, 8192), (32000, 4096)])
@pytest.mark.parametrize("draw", [torch.randn, torch.rand])
@pytest.mark.parametrize("M", [8, 3, 4])
def test_decode_rows_are_not_further_from_float64_than_the_exact_kernel(N, K, draw, M):
    """Operands of either sign and of one: what the tensor core cuts off when it adds must not add up.  Thousands of outputs each, so the
    2-norm errors are known to about half a percent; they lie two to twenty percent below those of the FMA kernel."""
    g = torch.Generator().manual_seed(N + K)
    fast = exact = 0.0
    for _ in range(3):
        x, w = draw(M, K, generator=g).bfloat16().cuda(), draw(N, K, generator=g).bfloat16().cuda()
        ref = x.double() @ w.double().T
        fast += float((SK.linear(x, w).double() - ref).norm() / ref.norm()) ** 2
        exact += float((SK.linear(x, w, tensor_cores=False).double() - ref).norm() / ref.norm()) ** 2
    assert fast <= exact


@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K", [(1, 8), (3, 2048), (130, 2056), (2371, 1024), (2371, 4096), (9481, 264), (600, 1528), (2368, 4096), (2372, 4096),
                                 (3000, 1024), (12000, 1024), (7200, 8192)])
def test_decode_rows_that_stay_give_the_same_bits(M, N, K, monkeypatch):
    """The kernel whose CTAs walk the features forms every sum in the order of the one with a CTA per four features (which batches take)."""
    g = torch.Generator().manual_seed(N + K + M)
    x, w = torch.randn(M, K, generator=g).bfloat16().cuda(), torch.randn(2, N, K, generator=g).bfloat16().cuda()
    want = torch.full((2 * M, N), 7.0, device="cuda")
    monkeypatch.setenv("JLLAMA_HYBRID_TC", "0")
    SK.linear_batched(torch.cat([x, x]), w, want, nbatch=2, rows=M, x_bs=M * K, o_bs=M * N)
    room = torch.full((M * N + 64,), 7.0, device="cuda")
    assert torch.equal(SK.linear(x, w[1], out=room[:M * N].view(M, N)), want[M:]) and bool((room[M * N:] == 7.0).all())
    check(SK.linear(x, w[0], act=SK.ACT_RELU, out_f32=False), x, w[0], torch.relu)


@pytest.mark.parametrize("M,K", [(1, 2048), (2, 1024), (4, 512)])
def test_decode_rows_of_a_parameter_in_a_graph(M, K):
    """A captured chain that asks for its weights ahead of the kernels before it sees the weights and tokens of every replay."""
    g = torch.Generator().manual_seed(K)
    x, w1, w2 = (torch.randn(s, K, generator=g).bfloat16().cuda() for s in (M, K, 777))

    def chain():
        return SK.linear(SK.linear(x, w1, out_f32=False, resident=True), w2, resident=True)

    chain()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = chain()
    for _ in range(3):
        graph.replay()
        y = SK.linear(x, w1, out_f32=False)
        assert torch.equal(out, SK.linear(y, w2))
        for t in (x, w1, w2):
            t.copy_(torch.randn(t.shape, generator=g).bfloat16())


@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K", [(2368, 2048), (2372, 3072), (2372, 3080), (3000, 4096), (2372, 2056), (3000, 1024)])
def test_early_and_late_decode_rows_have_the_same_bits(M, N, K):
    """Sizes on either side of the lines between the two kernels of up to four tokens, whose place depends on the early request; one of them forms the sums."""
    if K < 1536 or M < 3 or N < 3072:                       # (more features with 3 and 4 tokens: tensor cores)
        g = torch.Generator().manual_seed(N + K + M)
        x, w = torch.randn(M, K, generator=g).bfloat16().cuda(), torch.randn(N, K, generator=g).bfloat16().cuda()
        late, out = SK.linear(x, w), torch.full((M, N), 7.0, device="cuda")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            SK.linear(x, w, out=out, resident=True)
        graph.replay()
        assert torch.equal(out, late)
        check(late, x, w)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("K", [64, 77, 1024])
def test_a_single_row_of_any_pitch(dtype, K):
    """A column read as a row, a row repeated with pitch 0, the first row of a wide matrix: contiguous for torch, whatever the pitch of their one row says."""
    x, w = torch.randn(K, 1, device="cuda").to(dtype), torch.randn(96, K, device="cuda").to(dtype)
    want = SK.linear(x.view(1, K).clone(), w)
    wide = torch.randn(3, K + 5, device="cuda").to(dtype)
    wide[:1, :K] = x.t()
    for row in (x.t(), x.view(K).as_strided((1, K), (0, 1)), wide[:1, :K]):
        assert row.is_contiguous() and row.stride(0) != K and torch.equal(SK.linear(row, w), want)
