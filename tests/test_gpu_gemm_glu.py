"""Gated activations behind the tensor-core product, at the edges of its tiles, against float64."""
import pytest
import torch

from jax_llama_b200.config import DenseMlpSpec
from jax_llama_b200.models.feedforward import DenseFeedForward, _takes_gated_product
from jax_llama_b200.ops import _lib
from jax_llama_b200.ops import seq_kernels as SK

pytestmark = pytest.mark.gpu

ACTS = {"silu": lambda z: z * torch.sigmoid(z), "relu": torch.relu, "relu2": lambda z: torch.relu(z) ** 2,
        "gelu_tanh": lambda z: torch.nn.functional.gelu(z, approximate="tanh"), "sigmoid": torch.sigmoid, "none": lambda z: z,
        "xielu": lambda z: 0.5 * z}                        # (its two numbers are zero here)


@pytest.mark.parametrize("M", [1, 127, 128, 129, 300])
@pytest.mark.parametrize("F,Kd,gap", [(8, 8, 0), (120, 72, 16), (128, 64, 0), (136, 520, 8), (1000, 256, 0)])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh", "relu", "relu2", "sigmoid", "none", "xielu", "clamped"])
def test_gated_product(M, F, Kd, gap, act):
    """fp32 sums of K products (2^-17 of the sum of their sizes, tensor cores cut off when they add), fp32 activations, one rounding to bfloat16; nothing
    beyond the result is written."""
    g = torch.Generator().manual_seed(M + F + Kd)
    x, w = torch.randn(M, Kd, generator=g).bfloat16(), torch.randn(2 * F + gap, Kd, generator=g).bfloat16()
    gate, up = (x.double() @ w[o:o + F].double().T for o in (0, F + gap))
    size = [x.double().abs() @ w[o:o + F].double().abs().T for o in (0, F + gap)]
    if act == "clamped":
        a, b = gate.clamp(max=7.0), up.clamp(-7.0, 7.0)
        want = a * torch.sigmoid(1.702 * a) * (b + 1.0)
        kw, slope, outer = dict(kind=SK.GLU_CLAMPED, limit=7.0, alpha=1.702), 1.2, b.abs() + 1.0
        inner = a.abs()
    else:
        want = ACTS[act](gate) * up
        kw, slope, outer = dict(act=SK.ACTIVATIONS[act]), 1.2 if act != "relu2" else 2.0 * gate.abs().clamp(min=1.0), up.abs()
        inner = ACTS[act](gate).abs()
    got = SK.gemm_glu(x.cuda(), w.cuda(), F + gap, F, **kw).double().cpu()
    bound = 2.0 ** -8 * want.abs() + 2.0 ** -17 * (slope * size[0] * outer + size[1] * inner) + 1e-6
    assert bool(((got - want).abs() <= bound).all()), float(((got - want).abs() - bound).max())


@pytest.mark.parametrize("act", [SK.ACT_NONE, SK.ACT_RELU2, SK.ACT_SILU, SK.ACT_GELU_TANH, SK.ACT_SIGMOID, SK.ACT_RELU, SK.ACT_XIELU])
@pytest.mark.parametrize("N,Kd", [(8, 64), (264, 136), (512, 1024)])
def test_sorted_rows(N, Kd, act):
    """Tiles of several matrices, padding tiles, a device count that leaves the last tiles alone; the gated form over the same rows."""
    g = torch.Generator().manual_seed(N)
    x, w = torch.randn(640, Kd, generator=g).bfloat16().cuda(), (torch.randn(3, 2 * N, Kd, generator=g) * Kd ** -0.5).bfloat16().cuda()
    group, used = torch.tensor([2, 0, -1, 1, 1], dtype=torch.int32, device="cuda"), torch.tensor([4], dtype=torch.int32, device="cuda")
    for out_f32 in ((False, True) if act == SK.ACT_NONE else (False,)):
        got = SK.gemm_grouped(x, w, group, act=act, out_f32=out_f32, tiles_used=used)
        for t in (0, 1, 3):
            want = x[t * 128:(t + 1) * 128].double() @ w[int(group[t])].double().T
            if not out_f32:
                want = want.bfloat16().double()
                want = ACTS[next(n for n, a in SK.ACTIVATIONS.items() if a == act)](want)
            err = (got[t * 128:(t + 1) * 128].double() - want).abs()
            # a value that rounds the other way before the activation: two roundings, slope at most 2 max(1, |value|)
            assert bool((err <= (1e-4 if out_f32 else 2.0 ** -6 * (1.0 + want.abs()))).all())
    glu = SK.gemm_glu(x, w, N, N, act=SK.ACT_SILU, tile_group=group, tiles_used=used)
    for t in (0, 1, 3):
        a = x[t * 128:(t + 1) * 128].double()
        gate, up = a @ w[int(group[t]), :N].double().T, a @ w[int(group[t]), N:].double().T
        want = gate * torch.sigmoid(gate) * up
        assert bool(((glu[t * 128:(t + 1) * 128].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-3).all())


@pytest.mark.parametrize("M", [128, 129, 200, 256, 257])
@pytest.mark.parametrize("W,F,one", [(512, 1024, 201), (768, 1024, 257), (1024, 4736, 201), (2048, 2736, 257), (1024, 4744, 129), (504, 256, 129)])
def test_gated_layers_on_either_side_of_the_line(M, W, F, one):
    """Where product and activation are one kernel and where they are two: the gated values rounded to bfloat16 (2^-9 each), fp32 sums on both sides of
    them.  `one`: rows from which it is one."""
    g = torch.Generator(device="cuda").manual_seed(M + F)
    w = {n: (torch.randn(s, generator=g, device="cuda") * s[1] ** -0.5).bfloat16() for n, s in (("gate", (F, W)), ("up", (F, W)), ("down", (W, F)))}
    layer = DenseFeedForward(DenseMlpSpec(ff=F, act="silu", gated=True), w)
    h = torch.randn(M, W, generator=g, device="cuda").bfloat16()
    assert _takes_gated_product(h, layer.up, F) == (M >= one)
    d = {n: v.double() for n, v in w.items()}
    gate = h.double() @ d["gate"].T
    want = (gate * torch.sigmoid(gate) * (h.double() @ d["up"].T)) @ d["down"].T
    assert float((layer.run(h).double() - want).norm() / want.norm()) < 2.0 ** -8


@pytest.mark.parametrize("N", [8, 24])
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_sorted_rows_of_few_columns_at_any_element(N, f32, shift):
    """The C entry's result may start at any element where it has fewer than 32 columns; nothing around it is written."""
    Kd = 72
    g = torch.Generator().manual_seed(N)
    x, w = torch.randn(384, Kd, generator=g).bfloat16().cuda(), torch.randn(2, N, Kd, generator=g).bfloat16().cuda()
    group = torch.tensor([1, 0, 1], dtype=torch.int32, device="cuda")
    room = torch.full((384 * N + 16,), 7.0, dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
    out = room[shift:shift + 384 * N].view(384, N)
    _lib.check(_lib.lib().jl_gemm_grouped(x.data_ptr(), w.data_ptr(), out.data_ptr(), 384, N, Kd, 2, group.data_ptr(), 0, int(f32), 0,
                                          torch.cuda.current_stream().cuda_stream), "jl_gemm_grouped")
    want = torch.cat([x[t * 128:(t + 1) * 128].double() @ w[int(group[t])].double().T for t in range(3)])
    assert bool(((out.double() - want).abs() <= (1e-4 if f32 else 2.0 ** -8 * want.abs() + 1e-4)).all())
    assert bool((room[:shift] == 7.0).all()) and bool((room[shift + 384 * N:] == 7.0).all())
