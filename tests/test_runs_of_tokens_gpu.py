"""Kernels that take runs of tokens instead of single ones, alone, at the edges of their runs and blocks."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16}


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("channels,taps,offset", [(64, 4, 0), (66, 4, 2), (65, 4, 1), (1000, 8, 4), (20, 5, 0), (12, 1, 0), (516, 2, 8)])
def test_convolution_over_runs(cuda_device, dtype, channels, taps, offset):
    """Rows of 1 to 40 tokens over slots with inputs of their own, whose last inputs are then the slots'; channels that
    begin inside wider rows.  A tap's product is exact to a rounding; taps of them and the activation follow."""
    from zephyr_b200.kernels import ops

    g = torch.Generator().manual_seed(channels * 10 + taps)
    lengths, slots = [7, 1, 40, 8, 2, 17, 9], [3, 0, 6, 1, 5, 2, 4]
    T = sum(lengths)
    x = torch.randn(T, offset + channels + 3, generator=g).to(DTYPES[dtype]).to(cuda_device)[:, offset:offset + channels]
    w, bias = torch.randn(channels, taps, generator=g).to(cuda_device), torch.randn(channels, generator=g).to(cuda_device)
    state = torch.randn(8, (taps - 1) * channels + 1, generator=g).to(cuda_device)[:, :(taps - 1) * channels]
    before = state.clone()
    starts = [sum(lengths[:i]) for i in range(len(lengths))]
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)
    status = ops.new_status(cuda_device)
    out = ops.causal_conv_silu(x, channels, w, bias, state, i32(slots), i32(starts), i32(lengths),
                               i32([r for r, n in enumerate(lengths) for _ in range(n)]), status)
    ops.check_status(status)
    for start, n, slot in zip(starts, lengths, slots):
        inputs = torch.cat([before[slot].view(taps - 1, channels).double(), x[start:start + n].double()])
        z = sum(inputs[j:j + n] * w[:, j].double() for j in range(taps)) + bias.double()
        expected = z * torch.sigmoid(z)
        bound = 2.0 ** -22 * (taps + 4) if dtype == "float32" else 2.0 ** -8
        assert (out[start:start + n].double() - expected).abs().max() <= bound * max(1.0, float(expected.abs().max()))
        if taps > 1:
            assert torch.equal(state[slot].view(taps - 1, channels).double(), inputs[len(inputs) - taps + 1:])
