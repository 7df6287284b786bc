"""The weighted sum of the experts' rows (csrc/moe.cu): 16-byte columns against one float at a time, and both against float64."""
import pytest
import torch

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
