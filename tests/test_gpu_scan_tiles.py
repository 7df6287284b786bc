"""The prompt scans of the linear recurrences (csrc/gla_scan.cu) at the edges of their tiles, stages and time chunks, against float64.

S tokens of fp32 sums and products: every read-out is a sum over at most S tokens and D channels of products of decays, keys, values and
queries, each rounded a bounded number of times per token it passes; 2^-23 · (S + D) of the largest read-out bounds that by a wide margin, and
what a wrong tile, lane or chunk would leave is of the order of the read-out itself."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from jax_llama_b200.ops import seq_kernels as SK  # noqa: E402


@pytest.mark.parametrize("B,S,H,D,Dv", [(1, 9, 1, 10, 7), (2, 16, 3, 16, 64), (1, 17, 2, 33, 129), (3, 130, 1, 64, 128), (1, 700, 2, 64, 128),
                                        (2, 257, 2, 100, 36), (1, 200, 1, 128, 640), (1, 1000, 1, 256, 65), (2, 64, 40, 32, 64), (1, 333, 3, 17, 260)])
def test_projected_decays_over_a_prompt(B, S, H, D, Dv):
    g = torch.Generator().manual_seed(S * D + Dv)
    R = 5
    cols = 2 * H * D + H * Dv + R
    y = torch.randn(B * S, cols, generator=g)
    a2, bias = torch.randn(H * D, R, generator=g) * 0.5, 2.0 + torch.randn(H * D, generator=g)
    state = torch.randn(B, H, D, Dv, generator=g)
    pads = [0] + [min(S - 1, 5 + 21 * b) for b in range(1, B)]
    tau = 4.0
    want = torch.zeros(B, S, H, Dv, dtype=torch.float64)
    end = state.double().clone()
    yd = y.double().view(B, S, cols)
    q, k = yd[..., :H * D].reshape(B, S, H, D) * 0.25, yd[..., H * D:2 * H * D].reshape(B, S, H, D)
    v = yd[..., 2 * H * D:2 * H * D + H * Dv].reshape(B, S, H, Dv)
    alpha = torch.sigmoid(yd[..., -R:] @ a2.double().T + bias.double()).pow(1.0 / tau).view(B, S, H, D)
    for b in range(B):
        for t in range(pads[b], S):
            end[b] = alpha[b, t, :, :, None] * end[b] + k[b, t, :, :, None] * v[b, t, :, None]
            want[b, t] = torch.einsum("hdv,hd->hv", end[b], q[b, t])
    got_state = state.clone().cuda()
    got = SK.gla_scan(y.cuda(), 0, H * D, 2 * H * D, 2 * H * D + H * Dv, a2.cuda(), bias.cuda(), got_state,
                      torch.zeros(1, dtype=torch.int32, device="cuda"), torch.tensor(pads, dtype=torch.int32, device="cuda"), B, S, H, D, Dv, 0.25,
                      tau).double().cpu().view(B, S, H, Dv)
    tol = 2.0 ** -23 * (S + D)
    assert float((got - want).abs().max()) <= tol * float(want.abs().max())
    assert float((got_state.double().cpu() - end).abs().max()) <= tol * float(end.abs().max())


@pytest.mark.parametrize("R", [1536, 1537, 4000, 5900])
def test_wide_decay_projections(R):
    """Ranks whose rows of eight tokens outgrow the default shared memory (48 KB: 1536), up to what the staging check of the entry point
    leaves; the decays of a rank of thousands are summed in fp32 (2^-23 · R of their scale), everything after them as above."""
    B, S, H, D, Dv = 1, 21, 1, 16, 8
    g = torch.Generator().manual_seed(R)
    y = torch.randn(S, 2 * D + Dv + R, generator=g)
    a2, bias = torch.randn(D, R, generator=g) * R ** -0.5, torch.randn(D, generator=g)
    alpha = torch.sigmoid(y[:, -R:].double() @ a2.double().T + bias.double()).pow(0.25)
    state, want = torch.zeros(D, Dv, dtype=torch.float64), []
    for t in range(S):
        state = alpha[t][:, None] * state + y[t, D:2 * D].double()[:, None] * y[t, 2 * D:2 * D + Dv].double()
        want.append(state.T @ y[t, :D].double())
    want = torch.stack(want)
    end = torch.zeros(1, 1, D, Dv, device="cuda")
    got = SK.gla_scan(y.cuda(), 0, D, 2 * D, 2 * D + Dv, a2.cuda(), bias.cuda(), end, None, None, B, S, H, D, Dv, 1.0, 4.0).double().cpu()
    assert float((got - want).abs().max()) <= 2.0 ** -23 * (R + S + D) * float(want.abs().max())
    assert float((end.double().cpu()[0, 0] - state).abs().max()) <= 2.0 ** -23 * (R + S + D) * float(state.abs().max())


@pytest.mark.parametrize("S", [20, 700])                    # one chunk (the caller's state), several (the scratch)
@pytest.mark.parametrize("offset", [1, 2, 3])
def test_state_at_any_element(S, offset):
    """A state that starts off the 16-byte boundary gives the same numbers bit for bit."""
    B, H, D, Dv, R = 1, 2, 32, 64, 4
    g = torch.Generator().manual_seed(S + offset)
    y, a2, bias = torch.randn(S, 2 * H * D + H * Dv + R, generator=g).cuda(), torch.randn(H * D, R, generator=g).cuda(), torch.randn(H * D, generator=g).cuda()
    first = torch.randn(B, H, D, Dv, generator=g).cuda()
    room = torch.full((first.numel() + 8,), 7.0, device="cuda")
    moved = room[offset:offset + first.numel()].view_as(first)
    moved.copy_(first)
    scan = lambda state: SK.gla_scan(y, 0, H * D, 2 * H * D, 2 * H * D + H * Dv, a2, bias, state, None, None, B, S, H, D, Dv, 0.25, 4.0)
    want, got = scan(first), scan(moved)
    assert torch.equal(got, want) and torch.equal(moved, first)
    assert bool((room[:offset] == 7.0).all()) and bool((room[offset + first.numel():] == 7.0).all())


@pytest.mark.parametrize("dtype,ranks", [(torch.float32, (4, 12, 16, 20)), (torch.bfloat16, (8, 16, 24, 32, 40))])
@pytest.mark.parametrize("B,S,H,D,Dv", [(1, 9, 1, 10, 7), (2, 17, 3, 16, 64), (1, 130, 2, 33, 129), (3, 43, 5, 64, 30)])
def test_decay_projections_in_whole_pieces_match_the_general_preparation(dtype, ranks, B, S, H, D, Dv):
    """Ranks whose rows of A2 are whole 16-byte pieces, up to the instance's four and beyond; the same matrix off the boundary takes the
    general one.  The additions are the same ones in the same order: equal bit for bit."""
    for R in ranks:
        g = torch.Generator().manual_seed(S * D + R)
        y = torch.randn(B * S, 2 * H * D + H * Dv + R, generator=g).cuda()
        a2 = (torch.randn(H * D, R, generator=g) * 0.5).to(dtype).cuda()
        bias = torch.randn(H * D, generator=g).to(dtype).cuda()
        room = torch.zeros(a2.numel() + 1, dtype=dtype, device="cuda")
        off = room[1:].view(H * D, R)
        off.copy_(a2)
        pads = torch.tensor([0] + [3 + b for b in range(1, B)], dtype=torch.int32, device="cuda")
        first = torch.randn(B, H, D, Dv, generator=g).cuda()
        got, want = [], []
        for matrix, res in ((a2, got), (off, want)):
            state = first.clone()
            out = SK.gla_scan(y, 0, H * D, 2 * H * D, 2 * H * D + H * Dv, matrix, bias, state, torch.zeros(1, dtype=torch.int32, device="cuda"), pads,
                              B, S, H, D, Dv, 0.25, 4.0)
            res += [out, state]
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), R
        assert bool(torch.isfinite(got[0]).all())


@pytest.mark.parametrize("S", [1, 2, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("taps", [2, 4, 8, 31])
@pytest.mark.parametrize("pad", [0, 2])
def test_convolution_of_few_tokens(S, taps, pad):
    """Token counts on either side of the one from which several tokens are worked on side by side, against float64; the state afterwards, padding included."""
    g = torch.Generator().manual_seed(S + 100 * taps)
    B, C, off = 2, 130, 3
    y, w, bias = torch.randn(B * S, C + 5, generator=g), torch.randn(C, taps, generator=g), torch.randn(C, generator=g)
    state = torch.randn(B, taps - 1, C, generator=g)
    pads = torch.tensor([0, pad], dtype=torch.int32)
    x = y[:, off:off + C].reshape(B, S, C).double()
    for b in range(B):
        x[b, :int(pads[b])] = 0.0
    full = torch.cat([state.double(), x], 1)                                   # [B, taps - 1 + S, C]
    acc = bias.double() + sum(full[:, j:j + S] * w[:, j].double() for j in range(taps))
    want = acc * torch.sigmoid(acc)
    for b in range(B):
        want[b, :int(pads[b])] = 0.0
    kept = state.cuda()
    got = SK.causal_conv(y.cuda(), off, w.cuda(), bias.cuda(), kept, torch.zeros(1, dtype=torch.int32, device="cuda"), pads.cuda(), B, S, act=SK.ACT_SILU)
    assert float((got.view(B, S, C).double().cpu() - want).abs().max()) < 1e-5 * taps
    assert torch.equal(kept.cpu().double(), full[:, S:].float().double())
