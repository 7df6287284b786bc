"""Prompt attention of the generic head shapes on tensor cores (csrc/flash_wide.cu) against a float64 statement.

The inputs are bfloat16 and exact in float64; what the kernel rounds is a probability as hi + lo bfloat16 (2^-17 of it), fp32 sums, and the
output once to bfloat16 (2^-9 of a value): |error| <= 2^-8 |value| + 2^-14 of the largest value is twice what these give."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from jax_llama_b200.ops import seq_kernels as SK  # noqa: E402

F64 = torch.float64


def expected(q, k, v, scale, start, pads, window, chunk, sink, gate):
    """q [B, S, H, D]; k [B, T, G, D]; v [B, T, G, Dv] -> [B, S, H, Dv]."""
    B, S, H, D = q.shape
    T, G = k.shape[1], k.shape[2]
    i = torch.arange(start, start + S)[:, None]
    j = torch.arange(T)[None, :]
    out = torch.zeros(B, S, H, v.shape[-1], dtype=F64)
    for b in range(B):
        seen = (j <= i) & (j >= pads[b])
        if window:
            seen &= j > i - window
        if chunk:
            seen &= (j - pads[b]) // chunk == (i - pads[b]) // chunk
        for h in range(H):
            s = (q[b, :, h] @ k[b, :, h * G // H].T * scale).masked_fill(~seen, -math.inf)
            m = s.max(-1, keepdim=True).values.clamp_min(-1e30)
            e = torch.exp(s - m)
            den = e.sum(-1, keepdim=True)
            if sink is not None:
                den = torch.where(den > 0, den + torch.exp(sink[h] - m), den)
            out[b, :, h] = torch.where(den > 0, (e @ v[b, :, h * G // H]) / den.clamp_min(1e-300), 0.0)
            if gate is not None:
                out[b, :, h] *= torch.sigmoid(gate[b * S:(b + 1) * S, h:h + 1])
    return out


@pytest.mark.parametrize("D,Dv,B,S,start,T,H,G,window,chunk,extras,token_major", [
    (192, 128, 1, 129, 0, 129, 4, 4, 0, 0, False, True), (192, 128, 2, 300, 0, 300, 2, 2, 100, 0, True, True),
    (192, 64, 1, 2, 126, 140, 4, 2, 0, 0, False, False), (128, 128, 2, 64, 0, 64, 4, 1, 0, 0, True, False),
    (128, 64, 1, 65, 63, 200, 2, 1, 7, 0, False, False), (64, 128, 3, 63, 0, 63, 3, 3, 0, 50, True, True),
    (64, 64, 1, 257, 0, 257, 2, 2, 64, 0, False, False), (256, 128, 1, 200, 57, 257, 2, 1, 0, 64, False, False),
    (256, 64, 2, 31, 0, 31, 2, 2, 0, 0, True, True)])
def test_against_float64(D, Dv, B, S, start, T, H, G, window, chunk, extras, token_major):
    g = torch.Generator().manual_seed(D + S)
    bf = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)              # noqa: E731
    q, k, v = bf(B, S, H, D) * 2, bf(B, T, G, D), bf(B, T, G, Dv)
    pads = [(5 + 20 * b) % max(S, 2) for b in range(B)] if start == 0 else [11] * B
    sink = torch.randn(H, generator=g) if extras else None
    gate = torch.randn(B * S, H, generator=g) if extras else None
    scale = D ** -0.5
    want = expected(q.to(F64), k.to(F64), v.to(F64), scale, start, pads, window, chunk, None if sink is None else sink.to(F64),
                    None if gate is None else gate.to(F64))
    layout = {}
    if token_major:                                        # [B·T, G, d] rows, as a projection writes them
        kc, vc = k.cuda(), v.cuda()
        layout = dict(T_cap=T, ldk=G * D, ldv=G * Dv, strides=(T * G * D, D, T * G * Dv, Dv))
    else:                                                  # [B, G, T, d] caches
        kc, vc = k.transpose(1, 2).contiguous().cuda(), v.transpose(1, 2).contiguous().cuda()
    lens = torch.tensor([start], dtype=torch.int32, device="cuda")
    got = SK.attn_masked(q.reshape(B * S, H * D).contiguous().cuda(), kc, vc, lens, torch.tensor(pads, dtype=torch.int32, device="cuda"), B, S, H, G,
                         D, Dv, scale, gate=None if gate is None else gate.cuda(), window=window, chunk=chunk, sink=extras,
                         sink_logit=None if sink is None else sink.cuda(), **layout).double().cpu().view(B, S, H, Dv)
    assert bool(torch.isfinite(got).all())
    assert bool(((got - want).abs() <= 2 ** -8 * want.abs() + 2 ** -14 * want.abs().max()).all()), (got - want).abs().max()


def test_probabilities_keep_more_than_one_bfloat16():
    """Two keys whose values cancel: (p0 - p1) / (p0 + p1) of nearly equal probabilities is lost when they are rounded to 8 bits."""
    D, S = 128, 2
    q = torch.zeros(1, S, 1, D, dtype=torch.bfloat16)
    q[0, :, 0, 0] = 1.0
    k = torch.zeros(1, S, 1, D, dtype=torch.bfloat16)
    k[0, 1, 0, 0] = 2 ** -9                                 # scores 0 and 2^-9: p1 / p0 = 1.00195
    v = torch.ones(1, S, 1, 128, dtype=torch.bfloat16)
    v[0, 0] = -1.0
    want = math.tanh(2 ** -10)
    got = SK.attn_windowed(q.view(S, D).cuda(), k.transpose(1, 2).contiguous().cuda(), v.transpose(1, 2).contiguous().cuda(),
                           torch.zeros(1, dtype=torch.int32, device="cuda"), None, 1, S, 1, 1, D, 128, S, D, 128, 0, 1.0)
    assert abs(float(got[1, 0]) - want) <= 2 ** -6 * want   # one bfloat16 would give 0 or 2^-9, off by all of it


@pytest.mark.parametrize("D,Dv,B,S,start,T,H,G,window,chunk,token_major", [
    (192, 128, 1, 130, 0, 200, 2, 2, 0, 0, True), (192, 64, 2, 2, 126, 260, 4, 2, 0, 0, False), (128, 128, 2, 64, 0, 65, 4, 1, 0, 0, False),
    (128, 64, 1, 65, 70, 300, 2, 1, 7, 0, False), (64, 128, 3, 63, 0, 64, 3, 3, 0, 50, True), (64, 64, 1, 100, 3, 500, 2, 2, 64, 0, False),
    (256, 128, 1, 200, 57, 320, 2, 1, 0, 64, False), (256, 64, 2, 31, 0, 96, 2, 2, 0, 0, True)])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_slots_without_a_key_may_hold_anything(D, Dv, B, S, start, T, H, G, window, chunk, token_major, bad):
    """Behind the last key, before a row's first one, and before the first key that a window or chunk of the first tile reaches (64 slots of
    the tile at most): nothing of it reaches a result, which is bit for bit that of a clean cache."""
    g = torch.Generator().manual_seed(D + S)
    bf = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)              # noqa: E731
    q, k, v = bf(B, S, H, D).cuda(), bf(B, T, G, D).cuda(), bf(B, T, G, Dv).cuda()
    pads = torch.tensor([2 + b for b in range(B)], dtype=torch.int32)
    lo = pads.clone()                                       # first key that any query of the row sees
    if window:
        lo = torch.maximum(lo, torch.tensor(start - window + 1))
    if chunk:
        lo = torch.where(torch.tensor(start) >= pads, torch.maximum(lo, pads + (start - pads) // chunk * chunk), lo)
    lens = torch.tensor([start], dtype=torch.int32, device="cuda")

    def attend(k, v):
        layout = {}
        if token_major:
            layout = dict(T_cap=T, ldk=G * D, ldv=G * Dv, strides=(T * G * D, D, T * G * Dv, Dv))
        else:
            k, v = k.transpose(1, 2).contiguous(), v.transpose(1, 2).contiguous()
        return SK.attn_masked(q.reshape(B * S, H * D).contiguous(), k, v, lens, pads.cuda(), B, S, H, G, D, Dv, D ** -0.5, window=window, chunk=chunk,
                              **layout)
    clean = attend(k, v)
    slot = torch.arange(T)[None, :]
    dead = ((slot < lo[:, None]) | (slot >= start + S)).cuda()[:, :, None, None]
    got = attend(torch.where(dead, bad, k), torch.where(dead, bad, v))
    assert bool(torch.isfinite(clean).all()) and torch.equal(got, clean)


@pytest.mark.parametrize("D,Dv", [(64, 64), (128, 128), (192, 128), (256, 64)])
def test_a_nan_stays_visible(D, Dv):
    """A NaN or an infinite score is in the results of its own query and of no other; a query that sees no key stays zero."""
    B, S, H, T = 1, 150, 2, 150
    g = torch.Generator().manual_seed(D)
    q, k, v = (torch.randn(S, H, d, generator=g).to(torch.bfloat16).cuda() for d in (D, D, Dv))
    pads, lens = torch.tensor([3], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")

    def attend(q):
        return SK.attn_masked(q.reshape(S, H * D), k, v, lens, pads, B, S, H, H, D, Dv, D ** -0.5, T_cap=T, ldk=H * D, ldv=H * Dv,
                              strides=(T * H * D, D, T * H * Dv, Dv)).view(S, H, Dv)
    clean = attend(q)
    q[40, 1, 5] = float("nan")
    q[77, 0] = 3e38 * torch.sign(k[60, 0].float()).to(torch.bfloat16)              # its score with key 60 is +inf
    got = attend(q)
    assert bool(torch.isnan(got[40, 1]).all()) and bool(torch.isnan(got[77, 0]).all())
    same = torch.ones(S, H, dtype=torch.bool)
    same[40, 1] = same[77, 0] = False
    assert torch.equal(got[same.cuda()], clean[same.cuda()]) and bool((clean[:3] == 0).all())
