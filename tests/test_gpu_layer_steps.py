"""One token of a hybrid layer in one launch (jl_gla_step, jl_attn_step) beside the launches each stands in for, at the edges of their sizes.

Bound: both sides round the same stored quantities to bfloat16 (2^-9 of a value); the one launch keeps fp32 where the several store an intermediate, so a result
may fall one bfloat16 step (2^-8) another way, and fp32 sums in another order differ by 2^-20 of the largest term."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from jax_llama_b200.config import GlaMixerSpec, MoeMlpSpec  # noqa: E402
from jax_llama_b200.models.feedforward import MoeFeedForward  # noqa: E402
from jax_llama_b200.models.hybrid_engine import HybridCache  # noqa: E402
from jax_llama_b200.models.mixers import GlaMixer  # noqa: E402
from jax_llama_b200.ops import _lib  # noqa: E402
from jax_llama_b200.ops import kernels as K  # noqa: E402
from jax_llama_b200.ops import seq_kernels as SK  # noqa: E402


def i32(*v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def near(a, b, dtype):
    rel = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -18
    scale = float(b.abs().max())
    assert bool(((a.double() - b.double()).abs() <= rel * b.double().abs() + 2.0 ** -18 * scale).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,H,D,Dv,R", [(1, 1, 1, 1, 1), (2, 3, 64, 128, 16), (1, 2, 17, 33, 5), (3, 2, 128, 128, 16), (2, 2, 100, 64, 40), (1, 1, 32, 1000, 7), (1, 2, 256, 96, 9),
                                        (1, 2, 65, 500, 8)])
@pytest.mark.parametrize("weight", [True, False])
def test_gla_step(dtype, B, H, D, Dv, R, weight):
    g = torch.Generator(device="cuda").manual_seed(D * Dv + R)
    draw = lambda *n: torch.randn(*n, generator=g, device="cuda")        # noqa: E731
    y = draw(B, 2 * H * D + 2 * H * Dv + R + 3)
    offs = 0, H * D, 2 * H * D, 2 * H * D + 2 * H * Dv, 2 * H * D + H * Dv          # q, k, v, low-rank input, gate
    a2, bias, norm = (draw(H * D, R) * 0.3).to(dtype), (2 + draw(H * D)).to(dtype), draw(Dv).to(dtype) if weight else None
    state = draw(B, H, D, Dv)
    filled, pads = i32(9), i32(*[[0, 9, 10][b % 3] for b in range(B)])   # row 2: this token is padding
    other = state.clone()
    o = SK.gla_scan(y, *offs[:4], a2, bias, other, filled, pads, B, 1, H, D, Dv, 0.25, 8.0)
    if norm is not None:
        want = SK.headnorm_gate(o, norm, y[:, offs[4]:offs[4] + H * Dv], H, Dv, 1e-5, SK.ACT_SILU)
    else:
        r = torch.rsqrt(o.view(B, H, Dv).double().square().mean(-1, keepdim=True) + 1e-5)
        gate = y[:, offs[4]:offs[4] + H * Dv].double()
        want = ((o.view(B, H, Dv).double() * r).view(B, -1) * gate * torch.sigmoid(gate)).to(dtype)
    if not SK.gla_step_takes(D, Dv):
        with pytest.raises(RuntimeError):
            SK.gla_step(y, *offs, a2, bias, norm, state, filled, pads, B, H, D, Dv, 0.25, 8.0, 1e-5, SK.ACT_SILU)
        return
    got = SK.gla_step(y, *offs, a2, bias, norm, state, filled, pads, B, H, D, Dv, 0.25, 8.0, 1e-5, SK.ACT_SILU)
    near(got, want, dtype)
    assert torch.equal(state, other)                           # the state's update is the same arithmetic


@pytest.mark.parametrize("B,G,nkv,hd,T,filled,pads", [(1, 1, 1, 64, 16, 0, [0]), (2, 4, 4, 128, 90, 84, [0, 15]), (3, 2, 2, 64, 700, 699, [0, 300, 699]), (1, 8, 1, 128, 2000, 1500, [3]),
                                                      (2, 4, 2, 128, 600, 256, [0, 256]), (2, 1, 3, 128, 64, 10, [10, 11])])
@pytest.mark.parametrize("rot,unit,gate,own", [(64, True, True, True), (0, False, False, True), (32, True, True, False), (64, False, True, True)])
def test_attn_step(B, G, nkv, hd, T, filled, pads, rot, unit, gate, own):
    g = torch.Generator(device="cuda").manual_seed(B * T + hd)
    nh = G * nkv
    y = torch.randn(B, (nh + 2 * nkv) * hd + 8 + nh + nh % 2, generator=g, device="cuda")
    q_off, k_off, v_off, g_off = 2, 2 + nh * hd, 4 + (nh + nkv) * hd, 8 + (nh + 2 * nkv) * hd
    kc, vc = (torch.randn(B, nkv, T, hd, generator=g, device="cuda").bfloat16() for _ in range(2))
    half = max(rot // 2, 1)
    ang = torch.arange(T, device="cuda")[:, None] * 1000.0 ** (-torch.arange(half, device="cuda") / half)
    cos, sin = torch.cos(ang), torch.sin(ang)
    ln, pad = i32(filled), i32(*pads)
    k1, v1, k2, v2 = kc.clone(), vc.clone(), kc.clone(), vc.clone()
    q = torch.empty(B, nh * hd, dtype=torch.bfloat16, device="cuda")
    SK.attn_prep(y, q_off, k_off if own else -1, v_off if own else -1, q, k1 if own else None, v1 if own else None, cos, sin, rot, unit, 1e-5, ln, pad, B, 1, nh, nkv,
                 hd, hd)
    splits, scratch = K.decode_attn_plan(B, nh, nkv, hd, T, y.device)
    want = K.decode_attn(q.view(B, nh, hd), k1, v1, ln, pad, 1, splits, scratch)
    if gate:
        SK.head_gate(want, y[:, g_off:g_off + nh], nh, hd)
    got = torch.empty(B, nh * hd, dtype=torch.bfloat16, device="cuda")
    L = _lib.lib()
    _lib.check(L.jl_attn_step(y.data_ptr(), y.stride(0), q_off, k_off if own else -1, v_off if own else -1, g_off if gate else -1, cos.data_ptr(), sin.data_ptr(), T,
                              rot, int(unit), 1e-5, k2.data_ptr(), v2.data_ptr(), ln.data_ptr(), pad.data_ptr(), K._p(scratch), got.data_ptr(), B, nh, nkv, hd,
                              T, hd ** -0.5, splits, K._stream()), "jl_attn_step")
    # a head's rotated and scaled row may round to the other bfloat16 number (sums of squares in another order), nothing else of the caches changes
    near(k2, k1, torch.bfloat16)
    assert torch.equal(v2, v1)
    same = torch.ones(T, dtype=torch.bool, device="cuda")
    same[filled] = False
    assert torch.equal(k2[:, :, same], kc[:, :, same]) and torch.equal(v2[:, :, same], vc[:, :, same])
    scale = float(want.double().abs().max())
    assert float((got.double() - want.double()).abs().max()) <= 2.0 ** -7 * max(scale, 1e-6)


@pytest.mark.parametrize("splits", [1, 3])
def test_the_gates_exponential_is_not_approximated(splits):
    """One key whose values are ones: the result is the gate's sigmoid, rounded to bfloat16.  Computed to 2^-22 it can differ from the rounded exact one only where that lies
    within 2^-22 of the middle between two bfloat16 numbers; an exponential of the special-function unit is 2^-19 off at gates of -50: some of 65536 fall on the other side."""
    B, G, nkv, hd, T = 1024, 8, 8, 64, 8
    nh = G * nkv
    y = torch.ones(B, (nh + 2 * nkv) * hd + nh, device="cuda")
    y[:, -nh:] = torch.linspace(-80.0, 15.0, B * nh, device="cuda").view(B, nh)
    y[0, -3:] = torch.tensor([float("nan"), float("inf"), -float("inf")], device="cuda")
    kc, vc = (torch.zeros(B, nkv, T, hd, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    table, got = torch.zeros(1, 1, device="cuda"), torch.empty(B, nh * hd, dtype=torch.bfloat16, device="cuda")
    scratch = torch.empty(B * nh * splits * (hd + 2), device="cuda")
    L = _lib.lib()
    _lib.check(L.jl_attn_step(y.data_ptr(), y.stride(0), 0, nh * hd, (nh + nkv) * hd, (nh + 2 * nkv) * hd, table.data_ptr(), table.data_ptr(), 1, 0, 0, 1e-5, kc.data_ptr(),
                              vc.data_ptr(), i32(0).data_ptr(), i32(*[0] * B).data_ptr(), scratch.data_ptr(), got.data_ptr(), B, nh, nkv, hd, T, 1.0, splits,
                              K._stream()), "jl_attn_step")
    exact = torch.sigmoid(y[:, -nh:].double())[..., None].expand(B, nh, hd).reshape(B, -1)
    lo, hi = ((exact * (1 + e)).float().bfloat16() for e in (-2.0 ** -22, 2.0 ** -22))
    assert bool((((got >= lo) & (got <= hi)) | (got.isnan() & exact.isnan())).all()), int(((got < lo) | (got > hi)).sum()) // hd


def test_attn_step_refuses_rows_off_their_boundary():
    y = torch.randn(1, 999, device="cuda")
    L, p = _lib.lib(), y.data_ptr()
    assert L.jl_attn_step(p, 999, 0, 128, 256, -1, p, p, 4, 0, 0, 1e-5, p, p, 0, 0, 0, p, 1, 1, 1, 128, 4, 1.0, 1, K._stream()) != 0
    assert L.jl_attn_step(p, 998, 1, 128, 256, -1, p, p, 4, 0, 0, 1e-5, p, p, 0, 0, 0, p, 1, 1, 1, 128, 4, 1.0, 1, K._stream()) != 0


@pytest.mark.parametrize("M", [3, 20000])                      # intermediates that fit a room, and larger ones
def test_layers_derived_elsewhere_compute_with_tensors(M):
    """What a derived layer does with its base's intermediates is torch's to answer, whatever their size."""
    class Twice(GlaMixer):
        def run(self, h, B, S, cache, layer, rope=None):
            y = super().run(h, B, S, cache, layer, rope)
            return torch.cat([y[:, :7].float() * 2, 2 * y[:, 7:].float()], 1).to(y.dtype)

    class Shifted(MoeFeedForward):
        def _parts(self, h):
            args, more = super()._parts(h)
            return (args[0] + 1.0, *args[1:]), more

    g = torch.Generator(device="cuda").manual_seed(M)
    mat = lambda n, k: (torch.randn(n, k, generator=g, device="cuda") * k ** -0.5).bfloat16()        # noqa: E731
    W, H, D, Dv = 64, 2, 16, 32
    w = {"q": mat(H * D, W), "k": mat(H * D, W), "v": mat(H * Dv, W), "g": mat(H * Dv, W), "a1": mat(16, W), "a2": mat(H * D, 16), "a2.b": mat(1, H * D)[0], "norm": mat(1, Dv)[0],
         "o": mat(W, H * Dv)}
    h = mat(M, W)
    results = []
    for cls in (GlaMixer, Twice):
        m = cls(GlaMixerSpec(heads=H, dim=D, vdim=Dv, tau=16.0), w, 1e-5)
        cache = HybridCache(k=torch.zeros(1, device="cuda"), v=torch.zeros(1, device="cuda"), index=0, pad_left=i32(0), len_dev=i32(0), ks=[None], vs=[None],
                            states=[m.new_state(1, h.device)], length=M)
        results.append(m.forward(h, 1, M, cache, 0))
    assert torch.equal(results[1], 2 * results[0])             # a factor of two is exact
    ew = {"router": mat(4, W)}
    for e in range(4):
        ew[f"e{e}.gate"], ew[f"e{e}.up"], ew[f"e{e}.down"] = mat(24, W), mat(24, W), mat(W, 24)
    spec = MoeMlpSpec(experts=4, top=2, ff=24, act="silu", score="softmax", gated=True, shared_ff=0, shared_gate=False)
    plain, moved = MoeFeedForward(spec, ew).run(h), Shifted(spec, ew).run(h)
    assert float((moved - plain - 1.0).abs().max()) <= 2.0 ** -20 * float(plain.abs().max() + 1.0) * 4      # the weights of a token add up to one
