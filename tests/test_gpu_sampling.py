"""Exact full-vocabulary sampler (csrc/sample_full.cu) against the fp32 statement of the HF warper pipeline the
reference configures in jax_llama/generation.py:28-41 (temperature → top-k → top-p → categorical)."""
import itertools
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from jax_llama_b200.ops import kernels as K  # noqa: E402

V = 128256


def kept_set(logits, temperature, top_k, top_p):
    """Exact kept set and probabilities on the CPU in float64, ties ordered by lower index."""
    z = logits.double().cpu() / temperature
    order = torch.sort(z, descending=True, stable=True).indices          # stable: equal values keep index order
    if top_k and top_k < z.numel():
        order = order[:top_k]
    p = torch.softmax(z[order], 0)
    if top_p < 1.0:
        before = torch.cumsum(p, 0) - p
        order = order[before < top_p]
        p = torch.softmax(z[order], 0)
    return order, p


def test_argmax_picks_lowest_index_among_4096_tied_maxima():
    g = torch.Generator().manual_seed(0)
    x = torch.randn(3, V, generator=g)
    tied = torch.randperm(V, generator=g)[:4096]
    x[:, tied] = 9.0
    tok = K.sample_full(x.cuda(), temperature=0.0)
    assert tok.tolist() == [int(tied.min())] * 3


def test_constant_logits_top_k_keeps_the_lowest_indices():
    x = torch.zeros(V).cuda()
    tok = K.sample_full(x, temperature=1.0, top_k=5, seed=1, rows=4096)
    assert set(tok.tolist()) == {0, 1, 2, 3, 4}


@pytest.mark.parametrize("top_k,top_p,temperature,scale", [(0, 0.9, 0.8, 4.0), (100, 1.0, 1.0, 3.0), (1000, 0.95, 0.7, 1.0),
                                                           (0, 0.5, 1.0, 0.3)])
def test_samples_stay_inside_the_exact_nucleus_and_follow_its_distribution(top_k, top_p, temperature, scale):
    """No candidate budget: `top_k=None` is the nucleus over the whole vocabulary (flat logits keep tens of thousands of
    tokens), top_k = 100 / 1000 exceed any small candidate list."""
    g = torch.Generator().manual_seed(2)
    x = torch.randn(V, generator=g) * scale
    order, p = kept_set(x, temperature, top_k, top_p)
    n = 1 << 16
    tok = K.sample_full(x.cuda(), temperature=temperature, top_k=top_k, top_p=top_p, seed=7, rows=n).cpu().long()
    member = torch.zeros(V, dtype=torch.bool)
    member[order] = True
    assert bool(member[tok].all()), "a sampled token lies outside the exact kept set"
    # total variation between the empirical distribution and the exact one; the noise floor for `n` draws over `m`
    # atoms is about sqrt(m / (2 pi n))
    emp = torch.bincount(tok, minlength=V).double() / n
    exact = torch.zeros(V, dtype=torch.float64)
    exact[order] = p
    tv = 0.5 * (emp - exact).abs().sum().item()
    floor = (order.numel() / (6.28 * n)) ** 0.5
    assert tv < 1.5 * floor + 0.01, (tv, floor, order.numel())
    # the most likely token is sampled about as often as it should be
    top = int(order[0])
    assert abs(emp[top].item() - exact[top].item()) < 5 * (exact[top].item() / n) ** 0.5 + 1e-3


def test_same_seed_same_tokens_different_seed_different_tokens():
    x = (torch.randn(8, V, generator=torch.Generator().manual_seed(3)) * 2).cuda()
    step = torch.tensor([5], dtype=torch.int32, device="cuda")
    a = K.sample_full(x, temperature=0.9, top_k=50, top_p=0.9, seed=1, step=step)
    b = K.sample_full(x, temperature=0.9, top_k=50, top_p=0.9, seed=1, step=step)
    c = K.sample_full(x, temperature=0.9, top_k=50, top_p=0.9, seed=2, step=step)
    assert torch.equal(a, b) and not torch.equal(a, c)


def uniform_of(seed, step, row):
    """Philox-4x32-10 keyed by the seed at counter (step, row), as a number in (0, 1)."""
    m = 0xFFFFFFFF
    c = [step & m, row & m, 0x9E3779B9, 0xBB67AE85]
    k = [seed & m, (seed >> 32) & m]
    for _ in range(10):
        p0, p1 = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
        c = [(p1 >> 32) ^ c[1] ^ k[0], p1 & m, (p0 >> 32) ^ c[3] ^ k[1], p0 & m]
        k = [(k[0] + 0x9E3779B9) & m, (k[1] + 0xBB67AE85) & m]
    return ((c[0] >> 8) + 0.5) / 16777216.0


@pytest.mark.parametrize("rows,vocab,pitch,kind", [
    (1, 128256, 0, "normal"), (4, 128256, 0, "normal"), (30, 131072, 0, "normal"), (200, 8195, 1, "normal"), (3, 8191, 2, "normal"),
    (2, 8192, 0, "normal"), (5, 77, 3, "normal"), (2, 1, 0, "normal"), (3, 50001, 0, "coarse"), (2, 16384, 0, "plateau"), (4, 32003, 5, "masked"),
    (2, 40000, 0, "far")])
@pytest.mark.parametrize("top_k,top_p", [(0, 1.0), (0, 0.9), (300, 0.95), (7, 1.0)])
def test_tokens_are_the_inverse_cdf_of_the_kept_set(rows, vocab, pitch, kind, top_k, top_p):
    """Slices of one to eight CTAs, rows without 16-byte alignment, bins with many equal or neighbouring values, masked tokens."""
    g = torch.Generator().manual_seed(rows * vocab)
    x = torch.randn(rows, vocab + pitch, generator=g) * 3.0
    if kind == "coarse":
        x = (x * 2).round() / 2                            # a few dozen values, thousands of tokens on each
    elif kind == "plateau":
        x = x * 1e-4 + 50.0                                # everything within one bin, neighbouring floats
    elif kind == "masked":
        x[:, ::3] = float("-inf")
    elif kind == "far":
        x[:, 100:] -= 1000.0                               # most tokens have no mass: a large top-k reaches into them
    x = x.cuda()[:, :vocab]
    tok = K.sample_full(x, temperature=0.75, top_k=top_k, top_p=top_p, seed=12345678901, step=torch.tensor([9], dtype=torch.int32, device="cuda"))
    inv_temp = torch.tensor(1.0) / torch.tensor(0.75)       # the kernel's float32 scale
    for r in range(rows):
        z = (x[r].cpu() * inv_temp).double()
        order = torch.sort(z, descending=True, stable=True).indices
        if top_k and top_k < vocab:
            order = order[:top_k]
        p = torch.exp(z[order] - z.max())
        if top_p < 1.0:
            before = torch.cumsum(p, 0) - p
            # exponentials and fixed point differ from float64 by about 2^-21 of a mass: tokens that close to the cut may go either way
            sure = order[before < top_p * p.sum() * (1 - 2e-6)]
            order = order[before < top_p * p.sum() * (1 + 2e-6)]
            p = p[:order.numel()]
            lo_total, hi_total = p[:sure.numel()].sum().item(), p.sum().item()
        else:
            lo_total = hi_total = p.sum().item()
        u = uniform_of(12345678901, 9, r)
        edge = torch.cumsum(p, 0)
        i = int((order == int(tok[r])).nonzero().item())   # outside the kept set: no such element
        before, after = (edge[i] - p[i]).item(), edge[i].item()
        slack = 4e-6 * hi_total
        assert before <= u * hi_total + slack and after >= u * lo_total - slack, (r, u, before, after, hi_total)


@pytest.mark.parametrize("bad", ["nan", "inf", "all_masked"])
def test_rows_without_probabilities_still_give_a_token(bad):
    x = torch.randn(3, 20000, generator=torch.Generator().manual_seed(1)).cuda()
    if bad == "nan":
        x[1, 77] = float("nan")
    elif bad == "inf":
        x[1, 77] = float("inf")
    else:
        x[1] = float("-inf")
    y = K.sample_full(x, temperature=0.9, top_p=0.9, seed=3)
    assert bool(((y >= 0) & (y < 20000)).all())
    clean = K.sample_full(x[[0, 0, 2]].contiguous(), temperature=0.9, top_p=0.9, seed=3)
    assert y[0] == clean[0] and y[2] == clean[2]


@pytest.mark.parametrize("rows,vocab", [(1, 8192), (2, 8192), (1, 16385), (7, 32771), (12, 131072), (18, 8200)])
def test_clusters_exchange_their_best_after_all_of_them_have_started(rows, vocab):
    """Launches back to back, each starting under the tail of the one before it: the maximum moves through the slices of a row's CTAs, so a
    store into a CTA that has not begun, or a read before it, would give the token of an earlier launch."""
    x = torch.randn(rows, vocab, generator=torch.Generator().manual_seed(vocab)).cuda()
    at = [(i * vocab // 24 + 5 * i) % vocab for i in range(24)]
    inputs = []
    for a in at:
        y = x.clone()
        y[:, a] = 200.0
        inputs.append(y)
    greedy = [K.sample_full(y, temperature=0.0) for y in inputs]
    drawn = [K.sample_full(y, temperature=0.8, top_p=0.9, seed=1) for y in inputs]
    for a, t, u in zip(at, greedy, drawn):
        assert (t == a).all() and (u == a).all()


@pytest.mark.parametrize("first,second", [(1, 0), (255, 1), (128, 128), (128, 129), (256, 300), (257, 0), (90, 200)])
@pytest.mark.parametrize("vocab,skew", [(5000, 0), (20000, 3), (131072, 0)])
def test_answers_from_one_gather_and_from_several_agree_at_its_limit(first, second, vocab, skew):
    """Two plateaus one apart and nothing else: the boundaries of top-k, top-p and the draw fall into one bin or two, which hold up to 256 elements
    (one gather for all three) or more.  Within the plateaus every mass is known to 2^-21 of itself, so over at most 556 elements a sum is
    out by less than a thousandth of the smallest mass: the token's place in the order is the computed one or, next to an edge, its neighbour."""
    g = torch.Generator().manual_seed(first * 1000 + second)
    x = torch.full((3, vocab + skew), float("-inf"))
    orders = []
    for r in range(3):
        place = torch.randperm(vocab, generator=g)[:first + second]
        top, low = place[:first].sort().values, place[first:].sort().values
        x[r, top], x[r, low] = 2.0, 1.0
        orders.append(torch.cat([top, low]).tolist())
    dev = x.cuda()[:, :vocab]
    mass = [1.0] * first + [math.exp(-1.0)] * second
    for top_k, top_p in ((0, 1.0), (0, 0.6), (first + second // 2, 1.0), (first + second // 2, 0.9), (max(first // 2, 1), 0.3)):
        for seed in range(4):
            tok = K.sample_full(dev, temperature=1.0, top_k=top_k, top_p=top_p, seed=seed, step=torch.tensor([seed], dtype=torch.int32, device="cuda")).tolist()
            for r in range(3):
                kept = mass[:top_k] if top_k else mass
                edge = list(itertools.accumulate(kept))
                if top_p < 1.0:
                    edge = edge[:1 + sum(e < top_p * edge[-1] for e in edge)]
                want = sum(e <= uniform_of(seed, seed, r) * edge[-1] for e in edge)
                assert abs(orders[r].index(tok[r]) - want) <= 1, (top_k, top_p, seed, r)
