"""The delta rule in blocks at the edges of a block, of its halves and of a CTA's channels and value columns, against the rule in 64 bits."""

import pytest
import torch

from test_runs_of_tokens_gpu import _delta_in_float64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,groups,dim,vdim", [(3, 1, 64, 16), (2, 2, 65, 17), (6, 2, 128, 31)])
def test_blocks_are_near_the_rule_in_64_bits(cuda_device, dtype, heads, groups, dim, vdim):
    from zephyr_b200.kernels import ops

    lengths = [16, 17, 31, 32, 33, 48, 64, 65, 97]
    T, g = sum(lengths), torch.Generator().manual_seed(dim)
    q, k, v = (torch.randn(T, n, generator=g).to(dtype) for n in (groups * dim, groups * dim, heads * vdim))
    b, a = torch.randn(T, heads, generator=g), torch.randn(T, heads, generator=g)
    k[40:60] = k[40]                                       # one key twenty times over
    a_log, dt_bias, before = torch.randn(heads, generator=g), torch.randn(heads, generator=g) - 2.0, torch.randn(len(lengths), heads * dim * vdim, generator=g)
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)
    dev = lambda t: t.to(cuda_device)
    state, status, ba = dev(before), ops.new_status(cuda_device), dev(torch.cat([b, a], dim=1))
    starts = [sum(lengths[:i]) for i in range(len(lengths))]
    out = ops.delta_rule(dev(q), dev(k), dev(v), ba[:, :heads], ba[:, heads:], dev(a_log), dev(dt_bias), heads, groups, dim, vdim, state,
                         i32(list(range(len(lengths)))), i32(starts), i32(lengths), status, q_scale=dim ** -0.5, blocks_from=16)
    ops.check_status(status)
    for r, (start, n) in enumerate(zip(starts, lengths)):
        part = slice(start, start + n)
        expected, last = _delta_in_float64(q[part], k[part], v[part], b[part], a[part], a_log, dt_bias, heads, groups, dim, vdim, before[r])
        # Sums over the channels and the tokens before, in float32: the square root of their number of roundings of 2^-24 of values of
        # about one, a few times over along the chain from token to token.
        bound = 8 * (dim + n) ** 0.5 * 2.0 ** -24
        got = out[part].cpu().double().view_as(expected)
        assert (got - expected).norm() <= bound * expected.norm(), n
        assert (state[r].cpu().double().view_as(last) - last).norm() <= bound * last.norm(), n
