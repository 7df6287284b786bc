"""Decode attention on the tensor cores (csrc/decode_attn_fused.cu): blocks of keys through rings in shared memory, both head
widths, every group size, at the edges of blocks, splits and the cache, against the entry point's CPU statement."""
import pytest
import torch

from jax_llama_b200.models import reference as ref
from jax_llama_b200.ops import _lib, kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


# filled: none, one key, a block less / more one, a warp round, the last size that one CTA takes and the next, the cache full but one
@pytest.mark.parametrize("hd,filled,T", [(128, 0, 64), (128, 1, 64), (128, 15, 136), (128, 17, 136), (128, 65, 160), (128, 320, 1000), (128, 321, 1000),
                                         (128, 1999, 2000), (64, 31, 136), (64, 33, 136), (64, 129, 136), (64, 640, 1304), (64, 641, 1304),
                                         (64, 2047, 2048)])
@pytest.mark.parametrize("B,nkv,G", [(1, 1, 1), (1, 4, 8), (3, 4, 2), (20, 8, 4)])
def test_blocks_splits_and_cache_edges(B, nkv, G, hd, filled, T):
    nh = nkv * G
    g = torch.Generator().manual_seed(filled * 31 + B)
    rnd = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)
    qkv, kc, vc = rnd(B, (nh + 2 * nkv) * hd), rnd(B, nkv, T, hd), rnd(B, nkv, T, hd)
    cos, sin = ref.rope_cos_sin(hd, T, 500000.0)
    pad = torch.tensor([(7 * b * b) % max(filled, 1) for b in range(B)], dtype=torch.int32)
    clen = torch.tensor([filled], dtype=torch.int32)
    want = K.decode_attn_fused(qkv.float(), kc.float(), vc.float(), cos, sin, clen, pad, nh, nkv, hd)
    dead = torch.arange(T)[None, :] < pad[:, None]
    dead |= torch.arange(T)[None, :] > filled                 # slots that hold no key may hold anything
    gk, gv = (torch.where(dead[:, None, :, None], torch.tensor(float("nan"), dtype=torch.bfloat16), x).to(DEV) for x in (kc, vc))
    before = gk.clone(), gv.clone()
    splits, scratch = K.decode_attn_fused_plan(B, nh, nkv, hd, T, torch.device(DEV))
    K.set_decode_attn_variant(2)
    try:
        for _ in range(2):
            got = K.decode_attn_fused(qkv.to(DEV), gk, gv, cos.to(DEV), sin.to(DEV), clen.to(DEV), pad.to(DEV), nh, nkv, hd, splits, scratch)
    finally:
        K.set_decode_attn_variant(0)
    # rotated q and k are rounded to bfloat16 (2^-9 each: a score of size s moves by s * 2^-8, |s| <= ~6 here -> 2.4 % of a weight at
    # worst, averaged over the keys), the output once more (2^-9)
    got, want = got.float().cpu().view(B, nh, hd), want.view(B, nh, hd)
    assert torch.isfinite(got).all()
    err = (got - want).norm(dim=-1) / want.norm(dim=-1)
    assert err.max() < 3e-2 and err.mean() < 6e-3
    keep = torch.arange(T) != filled
    for now, was in zip((gk, gv), before):                    # nothing but the new slot was written
        assert torch.equal(now[:, :, keep.to(DEV)].view(torch.int16), was[:, :, keep.to(DEV)].view(torch.int16))
    assert torch.equal(gv[:, :, filled].cpu(), qkv.view(B, nh + 2 * nkv, hd)[:, nh + nkv:]) and (scratch[-B * nkv:] == 0).all()


@pytest.mark.parametrize("variant", [1, 2])
@pytest.mark.parametrize("hd,G", [(128, 4), (64, 1)])
@pytest.mark.parametrize("out_off,scratch_off", [(0, 0), (1, 0), (0, 1), (2, 3)])
def test_buffers_at_any_element(hd, G, out_off, scratch_off, variant):
    """The C entry takes an output and a scratch that start at any element; the merge uses wide accesses only where both allow it."""
    B, nkv, T, filled = 2, 4, 2048, 2000
    nh = nkv * G
    g = torch.Generator().manual_seed(hd)
    rnd = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16).to(DEV)
    qkv, kc, vc = rnd(B, (nh + 2 * nkv) * hd), rnd(B, nkv, T, hd), rnd(B, nkv, T, hd)
    cos, sin = (t.to(DEV) for t in ref.rope_cos_sin(hd, T, 500000.0))
    clen, pad = torch.tensor([filled], dtype=torch.int32, device=DEV), torch.zeros(B, dtype=torch.int32, device=DEV)
    splits, scratch = K.decode_attn_fused_plan(B, nh, nkv, hd, T, torch.device(DEV))
    assert splits > 1
    K.set_decode_attn_variant(variant)
    try:
        want = K.decode_attn_fused(qkv, kc.clone(), vc.clone(), cos, sin, clen, pad, nh, nkv, hd, splits, scratch)
        room = torch.zeros(scratch.numel() + 4, dtype=scratch.dtype, device=DEV)[scratch_off:scratch_off + scratch.numel()]
        out = torch.full((B * nh * hd + 8,), 7.0, dtype=torch.bfloat16, device=DEV)
        got = out[out_off:out_off + B * nh * hd].view(B, nh * hd)
        _lib.check(_lib.lib().jl_decode_attn_fused(qkv.data_ptr(), kc.data_ptr(), vc.data_ptr(), cos.data_ptr(), sin.data_ptr(), clen.data_ptr(),
                                                   pad.data_ptr(), room.data_ptr(), got.data_ptr(), B, nh, nkv, hd, T, T, hd ** -0.5, splits,
                                                   torch.cuda.current_stream().cuda_stream), "jl_decode_attn_fused")
    finally:
        K.set_decode_attn_variant(0)
    # the sums of the two merges run in the same order; a contraction may differ in the last bit of fp32, so one bfloat16 step at most
    torch.testing.assert_close(got.float(), want.float().view(B, nh * hd), rtol=2.0 ** -8, atol=2.0 ** -20)
    assert (out[:out_off] == 7.0).all() and (out[out_off + B * nh * hd:] == 7.0).all()
