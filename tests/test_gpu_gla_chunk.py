"""Prompt scans of the linear recurrences: with projected decays in chunks of 64 tokens on tensor cores (csrc/gla_chunk.cu) at the edges of their chunks, blocks and
tiles, with given decays token by token.

Oracle: the same scan token by token in float64, and for what is not finite the one-launch kernel of up to 8 tokens (csrc/gla_scan.cu), piece by piece.
Bound: every read-out is a sum over at most S tokens and D channels of products of decays, keys, values and queries, each rounded a bounded number
of times per token it passes; 2^-23 · (S + D) of the largest read-out bounds that by a wide margin, and a wrong tile, lane or chunk is of its order."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from jax_llama_b200.ops import seq_kernels as SK  # noqa: E402


def i32(*v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


class Gla:
    """Projected decays: y [B*S, q | k | v | z]."""
    tau = 4.0

    def __init__(self, B, S, H, D, Dv, R=16, seed=0):
        g = torch.Generator(device="cuda").manual_seed(seed + S * D + Dv)
        self.n = B, S, H, D, Dv
        self.cols = 2 * H * D + H * Dv + R
        self.y = torch.randn(B * S, self.cols, generator=g, device="cuda")
        self.a2, self.bias = torch.randn(H * D, R, generator=g, device="cuda") * 0.3, 2.0 + torch.randn(H * D, generator=g, device="cuda")
        self.state = torch.randn(B, H, D, Dv, generator=g, device="cuda")

    def scan(self, y, state, pads, filled=0, S=None):
        B, _, H, D, Dv = self.n
        S = self.n[1] if S is None else S
        o = SK.gla_scan(y, 0, H * D, 2 * H * D, 2 * H * D + H * Dv, self.a2, self.bias, state, i32(filled), i32(*pads), B, S, H, D, Dv, 0.25, self.tau)
        return o.view(B, S, H, Dv)

    def exact(self, pads, filled=0):
        B, S, H, D, Dv = self.n
        y = self.y.double().view(B, S, -1)
        q, k = y[..., :H * D].reshape(B, S, H, D) * 0.25, y[..., H * D:2 * H * D].reshape(B, S, H, D)
        v = y[..., 2 * H * D:2 * H * D + H * Dv].reshape(B, S, H, Dv)
        alpha = torch.sigmoid(y[..., 2 * H * D + H * Dv:] @ self.a2.double().T + self.bias.double()).pow(1.0 / self.tau).view(B, S, H, D)
        return exact_scan(q, k, v, alpha, self.state.double(), [max(0, p - filled) for p in pads])


def exact_scan(q, k, v, alpha, st, first):
    B, S, H, _ = q.shape
    o = torch.zeros(B, S, H, v.shape[-1], dtype=torch.float64, device="cuda")
    f = torch.tensor(first, device="cuda")
    for t in range(S):
        on = (t >= f).view(B, 1, 1, 1)
        st = torch.where(on, alpha[:, t, :, :, None] * st + k[:, t, :, :, None] * v[:, t, :, None], st)
        o[:, t] = torch.einsum("bhdv,bhd->bhv", st, q[:, t]) * on[:, :, 0]
    return o, st


def close(got, want, S, D):
    assert float((got.double() - want).abs().max()) <= 2.0 ** -23 * (S + D) * float(want.abs().max())


@pytest.mark.parametrize("B,S,H,D,Dv", [(1, 65, 1, 64, 128), (1, 127, 2, 10, 7), (2, 128, 3, 32, 64), (1, 129, 2, 33, 129), (3, 191, 1, 64, 128), (1, 192, 2, 65, 64),
                                        (2, 257, 2, 100, 36), (1, 700, 2, 128, 128), (1, 66, 1, 128, 260), (2, 640, 1, 1, 1), (1, 130, 40, 16, 24)])
def test_projected_decays(B, S, H, D, Dv):
    c = Gla(B, S, H, D, Dv)
    pads = [0] + [min(S - 1, 70 * b - 3) for b in range(1, B)]  # inside the second, third chunk: whole chunks of padding before
    state = c.state.clone()
    want, end = c.exact(pads)
    close(c.scan(c.y, state, pads), want, S, D)
    close(state, end, S, D)


@pytest.mark.parametrize("R", [1, 31, 32, 33, 70, 1537])
def test_ranks_of_the_decays(R):
    c = Gla(1, 70, 2, 20, 16, R=R)
    c.a2 *= R ** -0.5
    state = c.state.clone()
    want, end = c.exact([0])
    tol = 2.0 ** -23 * (R + 90)                                 # (the logits' sums of R terms beside the rest)
    got = c.scan(c.y, state, [0]).double()
    assert float((got - want).abs().max()) <= tol * float(want.abs().max()) and float((state.double() - end).abs().max()) <= tol * float(end.abs().max())


def test_a_prompt_that_continues_and_all_padding():
    c = Gla(2, 150, 2, 64, 64)
    state = c.state.clone()
    want, end = c.exact([5, 130], filled=20)                    # slots 20 ..: the padding of row 0 lies behind, 110 tokens of row 1 are padding
    close(c.scan(c.y, state, [5, 130], filled=20), want, 150, 64)
    close(state, end, 150, 64)
    state = c.state.clone()
    assert bool((c.scan(c.y, state, [400, 400]) == 0).all()) and torch.equal(state, c.state)


def test_values_state_and_rows_at_any_element():
    c = Gla(1, 140, 3, 64, 64)                                 # offsets of q, k, v off the 16-byte boundary, a pitch that is no multiple of four
    pads = [0]
    wide = torch.randn(140, c.cols + 3, device="cuda")
    wide[:, 1:1 + c.cols] = c.y
    room = torch.zeros(c.state.numel() + 1, device="cuda")
    moved = room[1:].view_as(c.state)
    moved.copy_(c.state)
    state = c.state.clone()
    B, S, H, D, Dv = c.n
    want = c.scan(c.y, state, pads)
    got = SK.gla_scan(wide, 1, 1 + H * D, 1 + 2 * H * D, 1 + 2 * H * D + H * Dv, c.a2, c.bias, moved, i32(0), i32(0), B, S, H, D, Dv, 0.25, 4.0)
    assert torch.equal(got.view_as(want), want) and torch.equal(moved, state)


@pytest.mark.parametrize("where", ["v", "k", "q", "z", "v inf", "k inf"])
def test_what_is_not_finite_stays_with_its_token_and_the_later_ones(where):
    c = Gla(1, 150, 2, 64, 64)
    clean_state = c.state.clone()
    clean = c.scan(c.y, clean_state, [0])
    H, D, Dv, t = 2, 64, 64, 83
    col = {"q": 5, "k": H * D + 70, "v": 2 * H * D + 9, "z": 2 * H * D + H * Dv + 2}[where[0]]
    c.y[t, col] = float("inf") if "inf" in where else float("nan")
    state, ref = c.state.clone(), c.state.clone()
    got = c.scan(c.y, state, [0])
    pieces = [c.scan(c.y[s:s + 8], ref, [0], S=min(8, 150 - s)) for s in range(0, 150, 8)]      # up to 8 tokens: one launch, token by token
    want = torch.cat(pieces, 1)
    assert torch.equal(got[:, :64], clean[:, :64])              # the chunk before is as it was, and nothing reaches an earlier token of its own
    assert bool(want[:, :t].isfinite().all()) and not bool(want.isfinite().all())
    for a, b in ((got, want), (state, ref)):
        fin = b.isfinite()
        assert torch.equal(a.isfinite(), fin) and torch.equal(a.isnan(), b.isnan())
        assert bool(((a - b).abs()[fin] <= 2.0 ** -23 * (150 + 64) * clean.abs().max()).all())


@pytest.mark.parametrize("layout,rot", [(SK.ROT_HALF, 64), (SK.ROT_INTERLEAVED, 32)])
def test_fixed_decays_with_rotation(layout, rot):
    B, S, H, D, Dv = 2, 200, 3, 64, 64
    g = torch.Generator(device="cuda").manual_seed(rot)
    y, state = torch.randn(B * S, 2 * H * D + H * Dv, generator=g, device="cuda"), torch.randn(B, H, D, Dv, generator=g, device="cuda")
    decay = torch.tensor([0.9, 0.99, 1.0], device="cuda")
    pos = torch.arange(S, device="cuda")
    ang = pos[:, None].double() * 1000.0 ** (-torch.arange(rot // 2, device="cuda").double() * 2 / rot)
    cos, sin = torch.cos(ang).float(), torch.sin(ang).float()
    pads = [0, 37]
    end = state.clone()
    got = SK.retention_scan(y, 0, H * D, 2 * H * D, decay, cos, sin, rot, layout, 0.25, end, i32(0), i32(*pads), B, S, H, D, Dv).view(B, S, H, Dv)

    def turn(z):
        z = z.clone()
        for b in range(B):
            p = (pos - pads[b]).clamp(min=0)
            cs, sn = cos[p].double()[:, None], sin[p].double()[:, None]
            a, e = (slice(0, rot, 2), slice(1, rot, 2)) if layout == SK.ROT_INTERLEAVED else (slice(0, rot // 2), slice(rot // 2, rot))
            u, v = z[b, ..., a].clone(), z[b, ..., e].clone()
            z[b, ..., a], z[b, ..., e] = u * cs - v * sn, v * cs + u * sn
        return z
    yd = y.double().view(B, S, -1)
    q, k = turn(yd[..., :H * D].reshape(B, S, H, D)), turn(yd[..., H * D:2 * H * D].reshape(B, S, H, D)) * 0.25
    alpha = decay.double().view(1, 1, H, 1).expand(B, S, H, D)
    want, st = exact_scan(q, k, yd[..., 2 * H * D:].reshape(B, S, H, Dv), alpha, state.double(), pads)
    close(got, want, S, D)
    close(end, st, S, D)


def test_the_exact_form_is_the_walk(monkeypatch):
    """JLLAMA_HYBRID_TC=0: fp32 FMAs token by token, shown by the state that pieces of 8 tokens leave (another kernel, the same roundings); the chunks on the tensor cores
    differ in the last bits."""
    S = 100                                                    # (too few tokens for chunks in time)
    c = Gla(2, S, 2, 64, 128)
    states = [c.state.clone() for _ in range(3)]
    a = c.scan(c.y, states[0], [0, 70])
    monkeypatch.setenv("JLLAMA_HYBRID_TC", "0")
    b = c.scan(c.y, states[1], [0, 70])
    for s in range(0, S, 5):
        c.scan(c.y.view(2, S, -1)[:, s:s + 5].reshape(10, -1).contiguous(), states[2], [0, 70], filled=s, S=5)
    assert torch.equal(states[1], states[2]) and not torch.equal(states[0], states[1]) and not torch.equal(a, b)
    want, _ = c.exact([0, 70])
    close(a, want, S, 64)
    close(b, want, S, 64)


@pytest.mark.parametrize("B,S,H,D,Dv", [(1, 65, 4, 64, 128), (2, 96, 4, 32, 64), (1, 500, 16, 64, 128), (4, 128, 16, 128, 128), (1, 2048, 4, 64, 128)])
@pytest.mark.parametrize("positive", [False, True])
@pytest.mark.parametrize("tau,bias", [(16.0, -1.0), (16.0, 2.0), (16.0, 8.0), (4.0, -1.0)])       # decays of 0.92, 0.99, 0.99998 and 0.72 in the mean
def test_error_beside_the_walk(B, S, H, D, Dv, positive, tau, bias, monkeypatch):
    """2-norms of the errors of read-outs and state are those of the walk in fp32 FMAs, whose decays have the same errors: 5 % above at most.  Two exceptions, as what the tensor
    core cuts off has a sign and the walk's roundings have none: states of one sign that forget within a chunk or two (20 %), and all of decays around 0.7, where sums have a
    few tokens (12 %, read-outs of one sign 40 %).  A chunk's sums in three of the six products are more than ten times off."""
    c = Gla(B, S, H, D, Dv)
    c.bias += bias - 2.0
    c.tau = tau
    if positive:
        c.y[:, :2 * H * D + H * Dv].abs_()
        c.state.abs_()
    want, end = c.exact([0] * B)
    errors = []
    for tc in ("1", "0"):
        monkeypatch.setenv("JLLAMA_HYBRID_TC", tc)
        state = c.state.clone()
        got = c.scan(c.y, state, [0] * B)
        errors.append((float((got.double() - want).norm()), float((state.double() - end).norm())))
    (o, st), (o_walk, st_walk) = errors
    few = tau == 4.0
    assert o <= (1.4 if few and positive else 1.12 if few else 1.05) * o_walk and st <= (1.2 if positive and bias < 0 else 1.12 if few else 1.05) * st_walk, (o / o_walk, st / st_walk)


@pytest.mark.parametrize("B,S,H,D,Dv", [(1, 64, 4, 64, 128), (2, 128, 2, 128, 64), (4, 60, 8, 32, 64)])
def test_a_chunks_state_of_one_sign(B, S, H, D, Dv):
    """Decays of exactly one, a state of zeros: sums of up to 128 products.  A sum of 16 is cut off by 3.3e-8 of it in the mean, three or four additions are rounded: 2^-24 · 5/4
    bounds them (measured 6.6e-8); all 64 in one sum are 9.8e-8 off."""
    c = Gla(B, S, H, D, Dv)
    c.y[:, :2 * H * D + H * Dv].abs_()
    c.bias += 60.0
    c.state.zero_()
    want, end = c.exact([0] * B)
    c.scan(c.y, c.state, [0] * B)
    assert float((c.state.double() - end).norm() / end.norm()) <= 1.25 * 2.0 ** -24


# What follows walks token by token (csrc/gla_scan.cu), in time chunks of its own: decays that are given need no fewer bits than fp32 additions have.

@pytest.mark.parametrize("B,S,H,D,Dv", [(1, 65, 4, 64, 128), (1, 500, 16, 64, 128), (1, 2048, 16, 64, 128), (4, 128, 16, 128, 128)])
@pytest.mark.parametrize("decay", [0.9, 1.0])
def test_fixed_decays_of_operands_of_one_sign(B, S, H, D, Dv, decay):
    """A read-out is a sum over D >= 64 channels whose roundings are independent and have no mean, so its error is little above its own rounding: at most 2^-24 of it in
    the mean (measured 4.1e-8 to 4.8e-8).  Sums that are cut off are 1.3e-7 away, products of 64 decays formed in advance 9e-8."""
    g = torch.Generator(device="cuda").manual_seed(S + D)
    y = torch.randn(B * S, 2 * H * D + H * Dv, generator=g, device="cuda").abs()
    state = torch.randn(B, H, D, Dv, generator=g, device="cuda").abs()
    yd, table = y.double().view(B, S, -1), torch.zeros(1, 1, device="cuda")
    q, k, v = yd[..., :H * D].reshape(B, S, H, D), yd[..., H * D:2 * H * D].reshape(B, S, H, D), yd[..., 2 * H * D:].reshape(B, S, H, Dv)
    dec = torch.full((H,), decay, device="cuda")
    want, _ = exact_scan(q, k, v, dec.double().view(1, 1, H, 1).expand(B, S, H, D), state.double(), [0] * B)
    got = SK.retention_scan(y, 0, H * D, 2 * H * D, dec, table, table, 0, 0, 1.0, state, i32(0), i32(*[0] * B), B, S, H, D, Dv).view_as(want)
    assert float((got.double() - want).norm() / want.norm()) <= 2.0 ** -24


@pytest.mark.parametrize("S", [65, 129, 700])
@pytest.mark.parametrize("H,G,D,Dv", [(4, 2, 64, 64), (3, 1, 128, 36), (2, 2, 10, 130)])
def test_state_space_scan(S, H, G, D, Dv):
    B = 2
    g = torch.Generator(device="cuda").manual_seed(S + D)
    rand = lambda *n: torch.randn(*n, generator=g, device="cuda")  # noqa: E731
    y, u = rand(B * S, H + 3), rand(B * S, 2 * G * D + H * Dv + 1)
    bias, a_log, state = rand(H) - 1.0, rand(H) * 0.5, rand(B, H, D, Dv)
    pads, end = [0, 64 + S // 70], state.clone()               # row 1: padding into the second chunk of 64
    got = SK.ssd_scan(y, 2, bias, a_log, u, 0, G * D, 2 * G * D, G, end, i32(0), i32(*pads), B, S, H, D, Dv).view(B, S, H, Dv)
    ud = u.double().view(B, S, -1)
    q, k = (ud[..., o:o + G * D].reshape(B, S, G, D).repeat_interleave(H // G, 2) for o in (0, G * D))
    dt = torch.nn.functional.softplus(y.double()[:, 2:2 + H].view(B, S, H) + bias.double())
    alpha = torch.exp(-torch.exp(a_log.double()) * dt)[..., None].expand(B, S, H, D)
    want, st = exact_scan(q, k, ud[..., 2 * G * D:2 * G * D + H * Dv].reshape(B, S, H, Dv) * dt[..., None], alpha, state.double(), pads)
    close(got, want, S, D)
    close(end, st, S, D)


@pytest.mark.parametrize("S", [65, 129, 700])
@pytest.mark.parametrize("H,D,Dv", [(2, 64, 127), (3, 32, 128), (2, 128, 60)])
def test_matrix_memory_scan(S, H, D, Dv):
    """The column of ones behind the values makes Dv + 1 of them; decays and scales as the gates' kernel gives them."""
    B = 2
    g = torch.Generator(device="cuda").manual_seed(S + D)
    y = torch.randn(B * S, 2 * H * D + H * Dv + 2 * H, generator=g, device="cuda")
    state, m_state = torch.randn(B, H, D, Dv + 1, generator=g, device="cuda"), torch.zeros(B, H, device="cuda")
    n, pads, end = 2 * H * D + H * Dv, [0, 64 + S // 70], state.clone()
    ib, fb = torch.zeros(H, device="cuda"), torch.full((H,), 2.0, device="cuda")
    got, aux = SK.mlstm_scan(y, 0, H * D, 2 * H * D, n, n + H, ib, fb, 15.0, 0.25, end, m_state, i32(0), i32(*pads), B, S, H, D, Dv)
    yd, aux = y.double().view(B, S, -1), aux.double().view(B, S, -1)
    q, k = yd[..., :H * D].reshape(B, S, H, D) * 0.25, yd[..., H * D:2 * H * D].reshape(B, S, H, D)
    v = torch.cat([yd[..., 2 * H * D:n].reshape(B, S, H, Dv), torch.ones(B, S, H, 1, dtype=torch.float64, device="cuda")], -1) * aux[..., H:2 * H, None]
    want, st = exact_scan(q, k, v, aux[..., :H, None].expand(B, S, H, D), state.double(), pads)
    close(got.view_as(want), want, S, D)
    close(end, st, S, D)
