"""Linear layers of the hybrid family at the sizes where their kernels change, against float64.

Products of the operands are formed exactly or in fp32 and summed in fp32: with K terms an error of a few 2^-24 of Σ |x w| per level of the
sum; 2^-20 Σ |x w| bounds every kernel here.  bfloat16 results add one rounding (2^-9)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from jax_llama_b200.ops import seq_kernels as SK  # noqa: E402


def check(got, x, w, act=lambda z: z):
    x, w = x.double(), w.double()
    ref = act(x @ w.T)
    bound = 2.0 ** -20 * (x.abs() @ w.abs().T) + (2.0 ** -8 if got.dtype == torch.bfloat16 else 2.0 ** -22) * ref.abs()
    assert bool(((got.double() - ref).abs() <= bound + 1e-30).all()), ((got.double() - ref).abs() - bound).max()


@pytest.mark.parametrize("M", [4, 5, 7, 8])
@pytest.mark.parametrize("N,K", [(1521, 2048), (1536, 8), (1543, 104), (4100, 264), (2048, 5464), (1600, 8200), (33000, 256)])
def test_decode_rows_bfloat16(M, N, K):
    g = torch.Generator().manual_seed(N + K + M)
    x, w = torch.randn(M, K, generator=g).bfloat16().cuda(), torch.randn(N, K, generator=g).bfloat16().cuda()
    check(SK.linear(x, w, tensor_cores=False), x, w)
    check(SK.linear(x, w, act=SK.ACT_RELU, out_f32=False), x, w, torch.relu)


def test_decode_rows_of_chosen_matrices():
    """One matrix per batch by index, some batches without one, several rows per batch."""
    g = torch.Generator().manual_seed(3)
    n, rows, N, K = 6, 6, 520, 392
    x, w = torch.randn(n * rows, K, generator=g).bfloat16().cuda(), torch.randn(4, N, K, generator=g).bfloat16().cuda()
    index = torch.tensor([2, -1, 0, 3, -1, 2], dtype=torch.int32, device="cuda")
    out = torch.full((n * rows, N), 7.0, device="cuda")
    SK.linear_batched(x, w, out, nbatch=n, rows=rows, x_bs=rows * K, o_bs=rows * N, w_index=index)
    for z, e in enumerate(index.tolist()):
        part = slice(z * rows, (z + 1) * rows)
        if e < 0:
            assert bool((out[part] == 7.0).all())
        else:
            check(out[part], x[part], w[e])
