"""float32 linears on CTA pairs (csrc/linear_f32_pair.cu) at the edges of their tiles, runs and sums, against float64.

Bound of an output, with A = sum |x w|: what the six products leave out (2^-24 A), what the tensor core cuts off (at most 2^-24 of the running sum at each
of the 24 steps of 64 k, so 24 · 2^-24 A), and the rounded additions of K / 64 sums, of the folds and of the parts (2^-24 A each)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from jax_llama_b200.ops import _lib  # noqa: E402
from jax_llama_b200.ops import seq_kernels as SK  # noqa: E402
from jax_llama_b200.ops.kernels import _stream, num_sms  # noqa: E402


def workspace(x, w):
    return _lib.lib().jl_linear_f32_pair_ws(x.data_ptr(), x.stride(0), w.data_ptr(), x.shape[0], w.shape[0], x.shape[1], num_sms(x.device))


def operands(M, N, K, seed=0, positive=False):
    g = torch.Generator(device="cuda").manual_seed(seed + M + N + K)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    return (x.abs(), w.abs()) if positive else (x, w)


def check(got, x, w):
    K = x.shape[1]
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    assert bool(((got.double() - want).abs() <= 2.0 ** -24 * (24 + 8 + K / 64) * size).all())


# rows at the edges of the tiles of 128, 192, 224 and 256; features and K off them; runs inside one tile, over several, whole tiles only; sums of more than 32 x 64 (the last: of
# whole tiles)
@pytest.mark.parametrize("M,N,K", [(65, 3000, 1024), (128, 2050, 1028), (129, 1024, 2048), (192, 4097, 260), (193, 1031, 1100), (200, 5464, 2048), (224, 1025, 2052),
                                   (225, 2048, 5464), (257, 256, 256), (300, 777, 256), (449, 512, 2116), (700, 257, 4228), (1025, 300, 300), (2000, 3001, 1024), (18944, 256, 4096)])
@pytest.mark.parametrize("positive", [False, True])
def test_against_float64(M, N, K, positive):
    x, w = operands(M, N, K, positive=positive)
    assert workspace(x, w) >= 0                                # these sizes run the kernel under test
    check(SK.linear(x, w), x, w)


# whole tiles; parts that meet in one or several tiles; sums of more than 32 x 64
@pytest.mark.parametrize("M,N,K", [(300, 256, 256), (400, 1600, 512), (200, 1100, 2048), (700, 257, 4228)])
def test_sums_that_need_no_rounding_are_exact(M, N, K):
    """One-hot rows and features (the one lies in every position of a block of 64 k, in even and odd blocks) give numbers back bit for bit; whole numbers whose
    sums stay below 2^24 add up exactly, with partial sums that cancel."""
    x, w = operands(M, N, K)
    hot = torch.zeros(M, K, device="cuda")
    at = torch.arange(M, device="cuda") * 61 % K
    hot[torch.arange(M, device="cuda"), at] = 1.0
    assert workspace(hot, w) >= 0
    assert torch.equal(SK.linear(hot, w), w[:, at].T)
    hot = torch.zeros(N, K, device="cuda")
    at = torch.arange(N, device="cuda") * 67 % K
    hot[torch.arange(N, device="cuda"), at] = 1.0
    assert torch.equal(SK.linear(x, hot), x[:, at])
    xi, wi = (x * 4).round(), (w * 4).round()
    assert torch.equal(SK.linear(xi, wi).double(), xi.double() @ wi.double().T)


@pytest.mark.parametrize("M,N,K", [(257, 256, 256), (300, 256, 256)])
def test_a_sum_that_one_pair_walks_alone_has_the_bits_of_the_single_ctas(M, N, K):
    x, w = operands(M, N, K)
    assert workspace(x, w) == 0                                # no runs that end inside a tile, no sums to fold
    single, L = torch.empty(M, N, device="cuda"), _lib.lib()
    _lib.check(L.jl_linear_any(x.data_ptr(), K, w.data_ptr(), single.data_ptr(), N, M, N, K, 0, 0.0, 0.0, 1, 1, _stream()), "jl_linear_any")
    assert torch.equal(SK.linear(x, w), single)


@pytest.mark.parametrize("M,N,K", [(300, 256, 256), (400, 1600, 512), (65, 3000, 1024), (200, 10928, 2048), (200, 2048, 5464), (1000, 1024, 1024), (200, 2048, 11000)])
@pytest.mark.parametrize("positive", [False, True])
def test_error_in_the_mean(M, N, K, positive):
    """2-norm of the error: 2^-23 of the result for what the six products leave out and the tensor core cuts off a block of 64 k (twice the 2^-24 that the latter
    measures), and sqrt(K / 64) / 4 · 2^-24 for the rounded additions.  Without the smallest of the six products normal operands give 2^-19."""
    x, w = operands(M, N, K, positive=positive)
    assert workspace(x, w) >= 0
    want = x.double() @ w.double().T
    assert float((SK.linear(x, w).double() - want).norm() / want.norm()) <= 2.0 ** -24 * (2.0 + (K / 64) ** 0.5 / 4)


@pytest.mark.parametrize("M,N,K", [(128, 10928, 2048), (200, 10928, 2048), (200, 10928, 4228), (200, 2048, 5464), (200, 2048, 11000), (400, 1600, 512), (2048, 6176, 1024)])
@pytest.mark.parametrize("positive", [False, True])
def test_error_is_not_above_the_single_ctas(M, N, K, positive):
    """Sums of as many blocks in a row at most: the same mean error, but for the sums that meet elsewhere (3 %)."""
    x, w = operands(M, N, K, positive=positive)
    assert workspace(x, w) >= 0
    single, L, want = torch.empty(M, N, device="cuda"), _lib.lib(), x.double() @ w.double().T
    _lib.check(L.jl_linear_any(x.data_ptr(), K, w.data_ptr(), single.data_ptr(), N, M, N, K, 0, 0.0, 0.0, 1, 1, _stream()), "jl_linear_any")
    assert float((SK.linear(x, w).double() - want).norm()) <= 1.03 * float((single.double() - want).norm())


def test_more_tiles_than_one_dimension_of_a_grid_takes():
    M, N, K = 524712, 8192, 512                                # 65600 tiles of 256 x 256 in runs that end inside tiles: 17 GB of results
    g = torch.Generator(device="cuda").manual_seed(5)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    assert workspace(x, w) > 0
    got = SK.linear(x, w)
    for rows in (slice(0, 300), slice(260000, 260300), slice(M - 300, M)):
        check(got[rows], x[rows], w)


def test_same_bits_again_and_inside_a_wider_result():
    x, w = operands(200, 1100, 2048)
    first = SK.linear(x, w)
    wide = torch.full((200, 1407), 7.0, device="cuda")
    SK.linear(x, w, out=wide[:, 101:1201])                     # an odd pitch and start
    assert torch.equal(wide[:, 101:1201], first)
    assert bool((wide[:, :101] == 7).all()) and bool((wide[:, 1201:] == 7).all())
    assert torch.equal(SK.linear(x, w), first)


def test_rows_of_a_wider_input():
    x, w = operands(150, 2048, 1024)
    wide = torch.randn(150, 1032, device="cuda")
    wide[:, 4:1028] = x
    assert torch.equal(SK.linear(wide[:, 4:1028], w), SK.linear(x, w))


@pytest.mark.parametrize("act,f", [(SK.ACT_RELU2, lambda z: torch.relu(z) ** 2), (SK.ACT_SILU, lambda z: z * torch.sigmoid(z))])
def test_activation(act, f):
    x, w = operands(140, 1100, 2048)
    assert workspace(x, w) >= 0
    z = SK.linear(x, w)
    got, want = SK.linear(x, w, act=act, out_f32=False).double(), f(z.double())
    assert float((got - want).abs().max()) <= 2.0 ** -20 * float(want.abs().max())


@pytest.mark.parametrize("M,N,K", [(300, 512, 512), (300, 777, 256), (200, 1100, 2048)])      # single CTAs; whole tiles; parts that meet
def test_not_finite_operands(M, N, K):
    """What is infinite or not a number in one row or feature stays there, as FMAs give it; finite operands above bfloat16's range too."""
    x, w = operands(M, N, K)
    plain = SK.linear(x, w)
    x[3, 5], x[17, K - 1], w[7, 9], w[30, 0], x[40, 70] = float("inf"), float("nan"), float("-inf"), float("nan"), 3.4e38
    got, want = SK.linear(x, w), SK.linear(x, w, tensor_cores=False)
    rows = torch.tensor([m for m in range(M) if m not in (3, 17, 40)], device="cuda")
    cols = torch.tensor([n for n in range(N) if n not in (7, 30)], device="cuda")
    assert torch.equal(got[rows][:, cols], plain[rows][:, cols])
    for a, b in ((got[[3, 17, 40]], want[[3, 17, 40]]), (got[:, [7, 30]], want[:, [7, 30]])):
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
        fin = b.isfinite()
        assert bool(((a - b).abs()[fin] <= 1e-3 * b.abs()[fin].clamp(min=1.0)).all())


def test_what_stays_with_the_other_kernels():
    for M, N, K in [(64, 4096, 1024), (128, 1024, 1024), (200, 512, 1024), (300, 255, 512), (300, 512, 252), (300, 512, 510), (300, 300, 512), (512, 256, 1024), (160, 512, 2048),
                    (65, 2048, 1024), (129, 1024, 1024), (140, 1100, 1024)]:
        x, w = operands(M, N, K)
        assert workspace(x, w) == -1
        check(SK.linear(x, w), x, w)
    room = torch.randn(300 * 512 + 1, device="cuda")
    x, w = room[1:].view(300, 512), torch.randn(512, 512, device="cuda")     # rows off the 16-byte boundary
    assert workspace(x, w) == -1
    check(SK.linear(x, w), x, w)
