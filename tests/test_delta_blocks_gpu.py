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


@pytest.mark.parametrize("dim,vdim", [(128, 20), (60, 16)])
def test_blocks_hold_values_up_to_the_largest_float32(cuda_device, dim, vdim):
    """A state's entry, and what a key writes, between the largest bfloat16 and the largest float32: read, carried and written as others are."""
    from zephyr_b200.kernels import ops

    heads, T, largest = 2, 80, torch.finfo(torch.float32).max
    g = torch.Generator().manual_seed(dim)
    q, k, v, b = (torch.randn(T, n, generator=g) for n in (dim, dim, heads * vdim, heads))
    a, a_log = torch.full((T, heads), -30.0), torch.zeros(heads)            # (next to no decay)
    before = torch.randn(heads, vdim, dim, generator=g)
    before[0, 1, 7], before[1, vdim - 1, dim - 1], before[0, 2, 30] = 3.395e38, -largest, 3.3999e38
    # Keys that see little of those entries keep them where they are; token 50 writes such a value of its own into the last column of head 0.
    k[:, [7, 30, dim - 1]] *= 1e-3
    k[50], b[50] = torch.nn.functional.one_hot(torch.tensor(3), dim).float(), 40.0
    v[50, vdim - 1] = 3.3999e38
    k[:, 3] *= (torch.arange(T) == 50).float()
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)
    dev = lambda t: t.to(cuda_device)
    state, status, ba = dev(before.reshape(1, -1)).clone(), ops.new_status(cuda_device), dev(torch.cat([b, a], dim=1))
    out = ops.delta_rule(dev(q), dev(k), dev(v), ba[:, :heads], ba[:, heads:], dev(a_log), torch.zeros(heads, device=cuda_device), heads, 1, dim, vdim,
                         state, i32([0]), i32([0]), i32([T]), status, q_scale=dim ** -0.5, blocks_from=16)
    ops.check_status(status)
    want, last = _delta_in_float64(q, k, v, b, a, a_log, torch.zeros(heads), heads, 1, dim, vdim, before)
    got, behind = out.cpu().double().view_as(want), state.cpu().double().view_as(last)
    assert last.abs().max() < largest and got.isfinite().all() and behind.isfinite().all()
    # Column by column, as a column's values do not meet another's: sums of float32 products along the chain of tokens.
    bound = 8 * (dim + T) ** 0.5 * 2.0 ** -24
    assert ((got - want).norm(dim=0) <= bound * want.norm(dim=0)).all()
    assert ((behind - last).norm(dim=2) <= bound * last.norm(dim=2)).all()
