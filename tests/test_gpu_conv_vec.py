"""Short convolutions of prompts, four channels a thread (csrc/seq_mix.cu causal_conv_vec_kernel), at the edges of their tokens and blocks.

Oracle: the walk that takes any alignment, asked for through columns off the 16-byte boundary; every sum is formed in the same order, so the bits are the
same."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from jax_llama_b200.ops import seq_kernels as SK  # noqa: E402


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,S,C", [(1, 9, 4), (2, 11, 36), (3, 12, 516), (1, 13, 1024), (2, 65, 132), (1, 1000, 2000), (1, 1001, 2004), (2, 999, 1004)])
@pytest.mark.parametrize("taps,act", [(1, SK.ACT_SILU), (2, SK.ACT_NONE), (3, SK.ACT_SILU), (4, SK.ACT_SILU), (4, SK.ACT_NONE)])
def test_same_bits_as_the_walk(dtype, B, S, C, taps, act):
    g = torch.Generator(device="cuda").manual_seed(S + C + taps)
    rand = lambda *n: torch.randn(*n, generator=g, device="cuda")  # noqa: E731
    x, w, bias, in_bias = rand(B * S, C), rand(C, taps).to(dtype), rand(C).to(dtype), rand(C)
    x[0, 0], x[-1, C - 1], x[S // 2, 1] = float("inf"), float("nan"), -float("inf")
    state = rand(B, taps - 1, C) if taps > 1 else None
    for filled, pads in ((0, [0, 5, S + 3][:B]), (7, [9, 0, 2][:B])):
        outs = []
        for col0 in (8, 9):
            y = torch.full((B * S, C + 12), 7.0, device="cuda")
            y[:, col0:col0 + C] = x
            st = state.clone() if taps > 1 else None
            out = SK.causal_conv(y, col0, w, bias, st, torch.tensor([filled], dtype=torch.int32, device="cuda"),
                                 torch.tensor(pads, dtype=torch.int32, device="cuda"), B, S, act=act, in_bias=in_bias)
            outs.append((out.view(torch.int32), st.view(torch.int32) if taps > 1 else out.view(torch.int32)))
        for a, b in zip(*outs):
            nan = torch.isnan(a.view(torch.float32))
            assert torch.equal(nan, torch.isnan(b.view(torch.float32))) and torch.equal(a[~nan], b[~nan])
