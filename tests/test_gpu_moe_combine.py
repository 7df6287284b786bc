"""The weighted sum of the experts' rows (csrc/moe.cu): 16-byte columns against one float at a time, and both against float64."""
import pytest
import torch

from jax_llama_b200.config import MoeMlpSpec
from jax_llama_b200.models.feedforward import MoeFeedForward
from jax_llama_b200.ops import seq_kernels as SK

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("W,pitch,shift", [(4, 4, 0), (1028, 1028, 0), (2048, 2056, 0), (2048, 2049, 0), (1030, 1030, 0), (1024, 1024, 1)])
@pytest.mark.parametrize("top", [1, 4, 8, 9])
@pytest.mark.parametrize("dtype,extras", [(torch.bfloat16, True), (torch.float32, True), (torch.bfloat16, False)])
def test_combine(W, pitch, shift, top, dtype, extras):
    """`pitch` and `shift` (floats) put the rows of z off the 16-byte boundary; nine experts take the general loop too."""
    M, R = 7, 80
    g = torch.Generator().manual_seed(W + top)
    flat = torch.randn(R * pitch + 4, generator=g).to(DEV)
    z = flat[shift:shift + R * pitch].view(R, pitch)[:, :W]
    pos = torch.randperm(R, generator=g)[:M * top].to(torch.int32).to(DEV)
    wt = torch.rand(M, top, generator=g).to(DEV)
    zz, ww = z.double()[pos.long()].view(M, top, W), wt.double()
    kw, shared, gate = {}, None, None
    if extras:
        shared, gate = torch.randn(M, W, generator=g).to(DEV), torch.randn(M, 1, generator=g).to(DEV)
        idx = torch.randint(0, 5, (M, top), generator=g).to(torch.int32)
        idx[::2, 0] = -1
        x = torch.randn(M, W, generator=g).to(dtype).to(DEV)
        ident = torch.rand(M, generator=g).to(DEV)
        kw = dict(idx=idx.to(DEV), ident_w=ident, x=x)
        ww = ww * (idx >= 0).to(DEV)
    want = (ww[..., None] * zz).sum(1)
    scale = (ww[..., None] * zz).abs().sum(1)
    if extras:
        want = want + ident.double()[:, None] * x.double() + torch.sigmoid(gate.double()) * shared.double()
        scale = scale + (ident.double()[:, None] * x.double()).abs() + shared.double().abs()
    got = SK.moe_combine(z, pos, wt, shared, gate, W, **kw)
    # top + 2 rounded additions and the gate's few roundings: (top + 2 + 4) * 2^-24 of the sum of magnitudes
    assert ((got.double() - want).abs() <= (top + 6) * 2.0 ** -24 * scale + 1e-30).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,experts,top", [(17, 32, 2), (40, 8, 1), (129, 32, 4), (300, 4, 2)])
def test_buffers_that_nobody_cleared_reach_no_result(M, experts, top, dtype, monkeypatch):
    """Few tokens and experts without any: whatever the uncleared buffers of the prompt path hold, the layer's output is the same bit for bit."""
    g = torch.Generator(device=DEV).manual_seed(M)
    W, F = 256, 136
    rnd = lambda *s: (torch.randn(*s, generator=g, device=DEV) * s[-1] ** -0.5).to(dtype)
    w = {"router": rnd(experts, W)}
    w["router"][experts // 2:] -= 1.0                          # positive inputs: the second half of the experts gets no token
    for e in range(experts):
        w[f"e{e}.gate"], w[f"e{e}.up"], w[f"e{e}.down"] = rnd(F, W), rnd(F, W), rnd(W, F)
    spec = MoeMlpSpec(experts=experts, top=top, ff=F, act="silu", score="softmax", gated=True, shared_ff=0, shared_gate=False)
    layer = MoeFeedForward(spec, w)
    h = torch.rand(M, W, generator=g, device=DEV).to(dtype)
    want = layer.run(h).clone()
    plain = torch.empty

    def poisoned(*a, **kw):
        t = plain(*a, **kw)
        return t.fill_(float("nan")) if t.is_floating_point() else t
    monkeypatch.setattr(torch, "empty", poisoned)
    got = layer.run(h)
    assert bool(torch.isfinite(want).all()) and torch.equal(got, want)


@pytest.mark.parametrize("M,top,E,tile", [(1, 1, 1, 16), (9, 4, 31, 16), (33, 3, 33, 64), (512, 2, 8, 16), (1025, 1, 8, 128), (1024, 4, 8, 128), (4097, 1, 6, 128),
                                            (2048, 4, 32, 128), (4096, 4, 300, 128), (4097, 4, 5, 128)])
@pytest.mark.parametrize("W", [8, 12, 2056])
def test_sorted_pairs_and_their_rows(M, top, E, tile, W):
    """Pairs a thread keeps in registers (one, four, sixteen) and more, rows on either side of the count up to which a CTA copies one, experts that do not divide among a warp's lanes, pairs without an expert; every
    pair's place lies in its expert's segment, the places are distinct, and the gathered rows are copies (zeros where no pair is)."""
    g = torch.Generator().manual_seed(M + E)
    idx = torch.randint(-1, E, (M, top), generator=g, dtype=torch.int32)
    pos, row_src, tile_group, used = (t.cpu() for t in SK.moe_sort(idx.cuda(), E, tile))
    flat = idx.flatten()
    counts = torch.bincount(flat[flat >= 0].long(), minlength=E)
    size = (counts + tile - 1) // tile * tile
    start = torch.cumsum(size, 0) - size
    assert int(used) == int(size.sum()) // tile
    assert tile_group[:int(used)].tolist() == torch.repeat_interleave(torch.arange(E), size // tile).tolist() and bool((tile_group[int(used):] == -1).all())
    real = flat >= 0
    assert bool((pos[~real] == -1).all())
    place, expert = pos[real].long(), flat[real].long()
    assert bool((place >= start[expert]).all()) and bool((place < start[expert] + counts[expert]).all()) and place.unique().numel() == place.numel()
    want = torch.full_like(row_src, -1)
    want[place] = (torch.arange(M * top, dtype=torch.int32) // top)[real]
    assert torch.equal(row_src, want)
    for dtype in (torch.bfloat16, torch.float32):
        x = torch.randn(M, W, generator=g).to(dtype)
        rows = torch.cat([x, torch.zeros(1, W, dtype=dtype)])[want.long()]
        for n in (len(want), max(1, len(want) - 1), max(1, len(want) - 3)):
            assert torch.equal(SK.moe_gather(x.cuda(), want[:n].cuda()).cpu(), rows[:n])


@pytest.mark.parametrize("M", [591, 592, 593])
@pytest.mark.parametrize("W,top", [(4, 1), (508, 3), (512, 8), (2052, 4)])
def test_threads_of_a_row_change_no_bit(M, W, top):
    """Rows on either side of the count from which a row has 128 threads: a column's sum is one thread's, in the order of the choices."""
    g = torch.Generator().manual_seed(M + W)
    z, wt, sh = torch.randn(M * top, W, generator=g), torch.rand(M, top, generator=g), torch.randn(M, W, generator=g)
    pos = torch.randperm(M * top, generator=g).int()
    d = [t.to(DEV) for t in (z, pos, wt, sh)]
    got = SK.moe_combine(*d, None, W)
    few = torch.cat([SK.moe_combine(d[0], d[1][i * top:(i + 100) * top], d[2][i:i + 100], d[3][i:i + 100], None, W) for i in range(0, M, 100)])
    want = (wt.double()[:, :, None] * z.double()[pos.long()].view(M, top, W)).sum(1) + sh.double()
    assert torch.equal(got, few)
    # top + 1 products and additions in fp32, each rounded once
    bound = 2.0 ** -23 * (top + 1) * ((wt[:, :, None] * z[pos.long()].view(M, top, W).abs()).sum(1) + sh.abs()).double()
    assert bool(((got.double().cpu() - want).abs() <= bound).all())
