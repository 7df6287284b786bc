"""Preparation of latent attention with 16-byte reads (csrc/attn_generic.cu latent_prep_vec_kernel) at the edges of what its registers hold, and beside it.

Oracle: the norms and the rotation in float64.  Bound: a sum of up to 2052 squares (2^-24 each, half of it in its root), the root, two products and the
rounding to the operand type: 2^-13 of the value in float32 is far above, 2^-8 in bfloat16 its rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from jax_llama_b200.ops import seq_kernels as SK  # noqa: E402


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("q_rank,normed", [(0, False), (4, True), (1024, True), (1028, True), (2048, True), (2052, True), (768, False), (30, True)])
@pytest.mark.parametrize("kv_rank,rot_dim", [(4, 0), (512, 64), (516, 8), (1024, 192), (1028, 4), (42, 6)])
def test_norms_rotation_and_append(dtype, q_rank, normed, kv_rank, rot_dim):
    g = torch.Generator(device="cuda").manual_seed(q_rank + kv_rank)
    rand = lambda *n: torch.randn(*n, generator=g, device="cuda")  # noqa: E731
    B, S, T, filled, pads = 2, 3, 9, 4, [0, 6]
    rot, kv_off = rot_dim // 4 * 2, (q_rank + 3) // 4 * 4
    y = rand(B * S, (kv_off + kv_rank + rot_dim + 7) // 4 * 4)
    wq, wkv = 1.0 + 0.3 * rand(max(q_rank, 4)).to(dtype), 1.0 + 0.3 * rand(kv_rank).to(dtype)
    angle = rand(T, max(rot // 2, 1))
    cos, sin = angle.cos(), angle.sin()
    cache = torch.full((B, T, kv_rank + rot_dim), 7.0, dtype=dtype, device="cuda")
    cq, c, kr = SK.latent_prep(y, 0, q_rank, kv_off, kv_rank, rot_dim, rot, 1, wq[:q_rank] if normed else None, wkv, cache, cos, sin, 1e-5,
                               torch.tensor([filled], dtype=torch.int32, device="cuda"), torch.tensor(pads, dtype=torch.int32, device="cuda"), B, S, True)
    tol = 2.0 ** -13 if dtype == torch.float32 else 2.0 ** -8

    def same(got, want):
        assert bool(((got.double() - want).abs() <= tol * want.abs() + 1e-6).all())

    norm = lambda x, w: x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w.double()  # noqa: E731
    d = y.double()
    if q_rank:
        same(cq, norm(d[:, :q_rank], wq[:q_rank]) if normed else d[:, :q_rank])
    want = norm(d[:, kv_off:kv_off + kv_rank], wkv)
    same(c, want)
    k = d[:, kv_off + kv_rank:kv_off + kv_rank + rot_dim].clone()
    if rot:
        pos = torch.tensor([max(0, filled + s - p) for p in pads for s in range(S)], device="cuda")
        co, si = cos.double()[pos], sin.double()[pos]
        u, v = k[:, :rot // 2].clone(), k[:, rot // 2:rot].clone()
        k[:, :rot // 2], k[:, rot // 2:rot] = u * co - v * si, v * co + u * si
    if rot_dim:
        assert bool(((kr.double() - k).abs() <= tol * k.abs() + 4e-6 * (1.0 + k.abs().max())).all())
        assert torch.equal(cache[:, filled:filled + S, kv_rank:].reshape(B * S, rot_dim), kr)
    assert torch.equal(cache[:, filled:filled + S, :kv_rank].reshape(B * S, kv_rank), c)
    assert bool((cache[:, :filled] == 7.0).all()) and bool((cache[:, filled + S:] == 7.0).all())
