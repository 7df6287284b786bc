"""The gated norm over parts of a row with 16-byte accesses (csrc/seq_mix.cu gated_groupnorm_vec_kernel) at the edges of its instances, and beside it.

Oracle: float64.  Bound: a sum of up to 4100 squares, an exponential, a root and a few products in float32, far inside 2^-13 of the value; bfloat16 rounds once (2^-8)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from jax_llama_b200.ops import seq_kernels as SK  # noqa: E402


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,groups,P", [(4, 1, 4), (512, 2, 64), (516, 1, 4), (1024, 2, 128), (1028, 3, 4), (2048, 1, 64), (2052, 1, 12), (4096, 1, 64), (4100, 1, 4), (30, 2, 6)])
@pytest.mark.parametrize("with_x", [True, False])
def test_parts_of_a_row(dtype, n, groups, P, with_x):
    g = torch.Generator(device="cuda").manual_seed(n)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    M, N = 5, n * groups
    o, z, w = rand(M, N), rand(M, N + 8)[:, 4:4 + N], (1.0 + 0.2 * rand(N)).to(dtype)
    x, skip = (rand(M, N + 4)[:, :N], rand(N // P).to(dtype)) if with_x else (None, None)
    got = SK.gated_groupnorm(o, x, skip, P, z, w, groups, 1e-5)
    v = o.double()
    if with_x:
        v = v + skip.double().repeat_interleave(P)[None] * x.double()
    inner = v.abs() if not with_x else o.double().abs() + (skip.double().repeat_interleave(P)[None] * x.double()).abs()
    gate = z.double() * torch.sigmoid(z.double())
    r = 1.0 / torch.sqrt(((v * gate).view(M, groups, n) ** 2).mean(-1, keepdim=True) + 1e-5)
    scale = (r.expand(M, groups, n).reshape(M, N) * w.double() * gate).abs()
    want = (v * gate).view(M, groups, n).mul(r).view(M, N) * w.double()
    tol = 2.0 ** -13 if dtype == torch.float32 else 2.0 ** -8
    assert bool(((got.double() - want).abs() <= tol * want.abs() + 2.0 ** -20 * inner * scale + 1e-7).all())
