"""The few-token GEMM (weights as the MMA's rows) at the edges of its tiles: token counts around multiples of 16 and its limits, ragged weight
rows and K, one tile, more tiles than two CTAs per SM hold at once, split and unsplit, outputs at any element."""
import pytest
import torch

from jax_llama_b200.ops import kernels as K
from jax_llama_b200.ops import seq_kernels as SK

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(M, N, Kd, seed):
    g = torch.Generator().manual_seed(seed)
    x, w, r = (torch.randn(s, generator=g).bfloat16() for s in ((M, Kd), (N, Kd), (M, N)))
    return x, (w.float() * Kd ** -0.5).bfloat16(), r


def _check(M, N, Kd, mode, shift=0):
    """Sums of K products in fp32 by a tensor core that cuts off when it adds (2^-17 of the sum of their sizes is four times what 5464 terms give), one
    rounding to bfloat16 per stored or intermediate value (2^-9 of it each, at most three in a row)."""
    K.ensure_gemm_workspace(torch.device(DEV))
    x, w, r = _inputs(M, N, Kd, M + N + Kd)
    xd, wd, rd = x.to(DEV), w.to(DEV), r.to(DEV)
    want = K.linear(xd.float().cpu().bfloat16(), w, residual=r if mode == "residual" else None, out_f32=mode == "f32",
                    mode={"residual": K.RESIDUAL, "swiglu": K.SWIGLU}.get(mode, K.PLAIN)).float()
    cols, dt = N // 2 if mode == "swiglu" else N, torch.float32 if mode == "f32" else torch.bfloat16
    buf = torch.full((M * cols + shift + 64,), 7.0, dtype=dt, device=DEV)
    out = buf[shift:shift + M * cols].view(M, cols)
    args = dict(out_f32=mode == "f32", out=out, force="gemm", mode={"residual": K.RESIDUAL, "swiglu": K.SWIGLU}.get(mode, K.PLAIN))
    if mode == "residual":
        args["residual"] = rd
    K.linear(xd, wd, **args)
    got = out.float().cpu()
    if mode == "f32":
        bound = 2.0 ** -17 * (x.float().abs() @ w.float().abs().T) + 1e-6
    else:
        bound = 3 * 2.0 ** -8 * (1.0 + want.abs())
    assert bool(((got - want).abs() <= bound).all()), float((got - want).abs().max())
    assert bool((buf[:shift] == 7.0).all()) and bool((buf[shift + M * cols:] == 7.0).all())
    first = out.clone()
    K.linear(xd, wd, **args)
    assert torch.equal(first, out)


@pytest.mark.parametrize("M", [5, 16, 17, 48, 49, 100, 112, 113, 128, 129, 160, 255, 256])
@pytest.mark.parametrize("N,Kd,mode", [(1000, 520, "plain"), (2048, 1024, "residual"), (4096, 2112, "swiglu"), (136, 256, "f32"),
                                       (11008, 4096, "plain")])
def test_token_counts(M, N, Kd, mode):
    _check(M, N, Kd, mode)


@pytest.mark.parametrize("M", [9, 33, 128])
@pytest.mark.parametrize("N,Kd,mode", [(128, 64, "plain"), (8, 8, "f32"), (18944, 192, "swiglu"), (19072, 320, "residual"), (37888, 128, "f32"),
                                       (38016, 200, "plain"), (50000, 128, "swiglu"), (4096, 16384, "residual"), (14336, 2048, "swiglu")])
def test_tile_counts(M, N, Kd, mode):
    _check(M, N, Kd, mode)


@pytest.mark.parametrize("M", [129, 130, 1000, 2048, 9472])
@pytest.mark.parametrize("N,Kd", [(8, 512), (32, 2048), (40, 520), (64, 1032)])
def test_few_features_over_many_tokens(M, N, Kd):
    _check(M, N, Kd, "f32")
    if M <= 4736:                                          # above, the token-major kernel, which stores 16 bytes at a time
        _check(M, N, Kd, "f32", shift=1)


@pytest.mark.parametrize("N,mode", [(32, "f32"), (40, "plain"), (64, "residual"), (264, "swiglu")])
def test_token_major_kernel_refuses_rows_off_the_16_byte_boundary(N, mode):
    """Results with a whole piece of 32 columns; narrower ones are stored element by element (below)."""
    x, w = torch.zeros(300, 64, dtype=torch.bfloat16, device=DEV), torch.zeros(N, 64, dtype=torch.bfloat16, device=DEV)
    cols, f32 = N // 2 if mode == "swiglu" else N, mode == "f32"
    room = torch.zeros(300 * cols + 8, dtype=torch.float32 if f32 else torch.bfloat16, device=DEV)
    out = room[1:1 + 300 * cols].view(300, cols)
    with pytest.raises(RuntimeError, match="16-byte"):
        K.linear(x, w, out_f32=f32, out=out, force="gemm", residual=torch.zeros_like(out) if mode == "residual" else None,
                 mode={"residual": K.RESIDUAL, "swiglu": K.SWIGLU}.get(mode, K.PLAIN))


@pytest.mark.parametrize("M", [129, 300, 4800])
@pytest.mark.parametrize("N,mode", [(8, "f32"), (24, "f32"), (16, "plain"), (24, "residual"), (16, "swiglu")])
def test_token_major_kernel_takes_narrow_results_at_any_element(M, N, mode):
    for shift in (0, 1):
        _check(M, N, 64, mode, shift)


@pytest.mark.parametrize("shift", [1, 2, 3])
@pytest.mark.parametrize("M,N,Kd", [(20, 1024, 2048), (20, 40000, 64)])
@pytest.mark.parametrize("mode", ["plain", "residual", "swiglu", "f32"])
def test_output_at_any_element(M, N, Kd, mode, shift):
    _check(M, N, Kd, mode, shift)


@pytest.mark.parametrize("M,N", [(16, 4096), (200, 4096), (2048, 32)])
def test_split_is_allowed_by_the_first_call_that_can_use_it(monkeypatch, M, N):
    """Whatever a process ran before: the permission is asked for at every size whose kernel may split K."""
    x, w = torch.zeros(M, 1024, dtype=torch.bfloat16, device=DEV), torch.zeros(N, 1024, dtype=torch.bfloat16, device=DEV)
    for call in (lambda: K.linear(x, w, out_f32=True), lambda: SK.linear(x, w)):
        monkeypatch.setattr(K, "_GEMM_WS", {})
        call()
        assert K._GEMM_WS


def _behind_their_writer(M, N, Kd, between, captured, rounds):
    """A norm writes the tokens, which held NaN, directly ahead of the product that reads them (with `between`, two kernels ahead, behind a
    product that lets the next kernel start before its own wait)."""
    K.ensure_gemm_workspace(torch.device(DEV))
    g = torch.Generator(device=DEV).manual_seed(M + N + Kd)
    xs = torch.randn(8, M, Kd, generator=g, device=DEV)
    gain = torch.ones(Kd, dtype=torch.bfloat16, device=DEV)
    w = (torch.randn(N, Kd, generator=g, device=DEV) * Kd ** -0.5).bfloat16()
    w2 = (torch.randn(512, Kd, generator=g, device=DEV) * Kd ** -0.5).bfloat16()
    h, x, out = torch.empty(M, Kd, dtype=torch.bfloat16, device=DEV), xs[0].clone(), torch.empty(M, N, device=DEV)
    out2 = torch.empty(M, 512, device=DEV)
    want = []
    for i in range(8):
        SK.norm_f32(xs[i], gain, 1e-5, 0.0, out=h)
        torch.cuda.synchronize()
        SK.linear(h, w, out=out)
        torch.cuda.synchronize()
        want.append(out.clone())

    def chain(src):
        h.fill_(float("nan"))
        SK.norm_f32(src, gain, 1e-5, 0.0, out=h)
        if between:
            SK.linear(h, w2, out=out2)
        SK.linear(h, w, out=out)

    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            chain(x)
    got = torch.empty(rounds, M, N, device=DEV)
    for r in range(rounds):
        if captured:
            x.copy_(xs[r % 8])
            graph.replay()
        else:
            chain(xs[r % 8])
        got[r].copy_(out)
    bad = [r for r in range(rounds) if not torch.equal(got[r], want[r % 8])]
    assert not bad, (len(bad), bad[:8])


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("M,N,Kd,between", [(129, 32, 2048, False), (200, 64, 512, True), (1000, 32, 2048, False), (2048, 8, 2048, False),
                                            (2048, 32, 2048, False), (2048, 64, 2048, False), (4096, 32, 1024, False), (4736, 32, 2048, False)])
def test_few_features_wait_for_the_kernel_that_writes_the_tokens(M, N, Kd, between, captured):
    _behind_their_writer(M, N, Kd, between, captured, 200)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("M,N,Kd,between", [(100, 2048, 2048, False), (128, 512, 2048, True), (200, 2048, 2048, False), (256, 4096, 1024, True)])
def test_few_tokens_wait_for_the_kernel_that_writes_them(M, N, Kd, between, captured):
    _behind_their_writer(M, N, Kd, between, captured, 100)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("M,N,Kd", [(129, 2048, 2048), (200, 512, 4096), (256, 4096, 1024)])
def test_weights_of_more_than_128_tokens_may_be_a_kernels_result(M, N, Kd, captured):
    """A cast writes the weights, which held NaN, directly ahead of the product."""
    K.ensure_gemm_workspace(torch.device(DEV))
    g = torch.Generator(device=DEV).manual_seed(M + N)
    masters = torch.randn(4, N, Kd, generator=g, device=DEV) * Kd ** -0.5
    x = torch.randn(M, Kd, generator=g, device=DEV).bfloat16()
    w, master, out = torch.empty(N, Kd, dtype=torch.bfloat16, device=DEV), masters[0].clone(), torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    want = [K.linear(x, m.bfloat16()) for m in masters]

    def chain(src):
        w.fill_(float("nan"))
        SK.act_cast(src, torch.bfloat16, out=w)
        K.linear(x, w, out=out)

    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            chain(master)
    for r in range(100):
        if captured:
            master.copy_(masters[r % 4])
            graph.replay()
        else:
            chain(masters[r % 4])
        assert torch.equal(out, want[r % 4])


def test_kernels_that_share_tensor_memory_take_turns():
    """Products with little shared memory, so that the next one's CTAs come to the same SMs, before products that take all columns of tensor memory."""
    K.ensure_gemm_workspace(torch.device(DEV))
    g = torch.Generator(device=DEV).manual_seed(1)
    few, many = torch.randn(16, 64, generator=g, device=DEV).bfloat16(), torch.randn(300, 64, generator=g, device=DEV).bfloat16()
    w = (torch.randn(20000, 64, generator=g, device=DEV) / 8).bfloat16()
    want_few, want_many = (few.double() @ w.double().T), (many.double() @ w[:2048].double().T)
    out_few, out_many = torch.empty(16, 20000, device=DEV), torch.empty(300, 2048, device=DEV)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(50):
            K.linear(few, w, out=out_few, out_f32=True)
            K.linear(many, w[:2048], out=out_many, out_f32=True)
    for _ in range(10):
        graph.replay()
    torch.cuda.synchronize()
    assert float((out_few.double() - want_few).abs().max()) < 1e-4 and float((out_many.double() - want_many).abs().max()) < 1e-4
