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


def test_the_delta_rule_on_both_paths(cuda_device):
    """A step whose rows bring runs goes block by block, single tokens one by one: a request cut either way ends in the
    same outputs and the same state, also where keys repeat (the block's matrix is then far from the unit matrix) and
    where a decay is so strong that a block forgets its start."""
    from zephyr_b200.kernels import ops

    heads, groups, dim, vdim, T = 4, 2, 128, 128, 83
    g = torch.Generator().manual_seed(5)
    q, k, v = (torch.randn(T, n, generator=g).to(cuda_device) for n in (groups * dim, groups * dim, heads * vdim))
    k[20:40] = k[20]                                       # one key twenty times over
    ba = (torch.randn(T, 2 * heads, generator=g) * 1.5).to(cuda_device)
    ba[50:53, heads:] = 60.0                               # decays of e^-60 and less
    a_log, dt_bias = (torch.randn(heads, generator=g) * 0.5).to(cuda_device), torch.zeros(heads, device=cuda_device)
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)
    status = ops.new_status(cuda_device)

    def run(cuts):
        state, out, at = torch.zeros(1, heads * dim * vdim, device=cuda_device), [], 0
        for n in cuts:
            part = slice(at, at + n)
            out.append(ops.delta_rule(q[part], k[part], v[part], ba[part, :heads], ba[part, heads:], a_log, dt_bias, heads, groups,
                                      dim, vdim, state, i32([0]), i32([0]), i32([n]), status, q_scale=dim ** -0.5))
            at += n
        ops.check_status(status)
        return torch.cat(out), state

    assert ops.DELTA_BLOCKS_FROM <= 17
    single, blocks, mixed = run([1] * T), run([T]), run([17, 3, 30, 1, 32])
    for other in (blocks, mixed):
        for x, y in zip(single, other):       # float32 sums in another order
            assert (x - y).abs().max() <= 1e-5 * max(1.0, float(x.abs().max()))
