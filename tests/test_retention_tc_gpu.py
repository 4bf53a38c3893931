"""Retention's walk in pieces of 128 tokens at the edges of a piece, of a head's channels and of a CTA's value columns, against the recurrence
in 64 bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,dim,vdim,rot", [(3, 128, 64, 128), (2, 100, 68, 64), (5, 68, 4, 0), (40, 128, 128, 64)])
def test_pieces_are_near_the_recurrence_in_64_bits(cuda_device, heads, dim, vdim, rot):
    from zephyr_b200.kernels import ops

    lengths, order = [127, 1, 128, 129, 64, 300], [2, 0, 5, 1, 4, 3]      # (rows may lie in the stream in any order)
    T, g = sum(lengths), torch.Generator().manual_seed(dim)
    starts, at = [0] * len(lengths), 0
    for r in order:
        starts[r], at = at, at + lengths[r]
    projected = torch.randn(T, heads * (2 * dim + vdim), generator=g).to(cuda_device)
    q, k, v = projected.split([heads * dim, heads * dim, heads * vdim], dim=1)
    decay = torch.rand(heads, generator=g).clamp(0.05, 0.999).to(cuda_device)
    decay[0] = 0.0
    positions = torch.zeros(T, dtype=torch.int32, device=cuda_device)
    for start, n in zip(starts, lengths):
        positions[start:start + n] = torch.arange(7, 7 + n)
    before = torch.randn(len(lengths), heads * dim * vdim, generator=g).to(cuda_device)
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)
    freqs = torch.rand(rot // 2, generator=g).to(cuda_device) if rot else None
    turn = dict(freqs=freqs, rot_dims=rot, k_scale=0.5, positions=positions) if rot else {}
    state, status, launched = before.clone(), ops.new_status(cuda_device), ops.LAUNCH_COUNTS.get("retention_tc", 0)
    out = ops.retention(q, k, v, decay, heads, dim, vdim, state, i32(list(range(len(lengths)))), i32(starts), i32(lengths), status, **turn)
    ops.check_status(status)
    assert ops.LAUNCH_COUNTS.get("retention_tc", 0) == launched + 2
    qd, kd, vd = q.double().view(T, heads, dim), k.double().view(T, heads, dim), v.double().view(T, heads, vdim)
    if rot:
        angle = (positions.float().unsqueeze(1) * freqs).double().unsqueeze(1)
        c, s, half = angle.cos(), angle.sin(), rot // 2
        turned = lambda x: torch.cat([x[..., :half] * c - x[..., half:rot] * s, x[..., half:rot] * c + x[..., :half] * s, x[..., rot:]], dim=-1)
        qd, kd = turned(qd), turned(kd) * 0.5
    for r, (start, n) in enumerate(zip(starts, lengths)):
        S, expected = before[r].double().view(heads, dim, vdim), []
        for t in range(start, start + n):
            S = S * decay.double().view(-1, 1, 1) + kd[t].unsqueeze(-1) * vd[t].unsqueeze(1)
            expected.append((qd[t].unsqueeze(-1) * S).sum(1))
        # Two bfloat16 parts leave an operand 2^-17 of itself away, in random directions; up to four of them stand behind an output.
        bound = 4 * 2.0 ** -17
        got, want = out[start:start + n].double().view(n, heads, vdim), torch.stack(expected)
        assert (got - want).norm() <= bound * want.norm(), n
        assert (state[r].double().view_as(S) - S).norm() <= bound * S.norm(), n


@pytest.mark.parametrize("dim,vdim", [(128, 128), (100, 68)])
def test_a_value_that_is_not_finite_stays_with_later_tokens(cuda_device, dim, vdim):
    """Infinities, NaN and values that round to infinity in bfloat16 among the values, at the edges of pieces, of the weights' quarters and of a
    CTA's columns, also in pieces that follow one another: all tokens before one, and all other columns, keep their bits."""
    from zephyr_b200.kernels import ops

    heads, T = 3, 300
    g = torch.Generator().manual_seed(dim)
    q, k, v = (torch.randn(T, n, generator=g).to(cuda_device) for n in (heads * dim, heads * dim, heads * vdim))
    decay, status = torch.tensor([0.4, 0.9, 0.999], device=cuda_device), ops.new_status(cuda_device)
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)

    def run(values):
        state, launched = torch.zeros(1, heads * dim * vdim, device=cuda_device), ops.LAUNCH_COUNTS.get("retention_tc", 0)
        out = ops.retention(q, k, values, decay, heads, dim, vdim, state, i32([0]), i32([0]), i32([T]), status)
        ops.check_status(status)
        assert ops.LAUNCH_COUNTS["retention_tc"] == launched + 2
        return out, state.view(heads, dim, vdim)

    clean, behind = run(v)
    inf, nan = float("inf"), float("nan")
    cases = [{(0, 0): nan}, {(31, 63): inf}, {(32, 64): -inf}, {(127, vdim - 1): nan}, {(128, vdim): inf}, {(299, 3 * vdim - 1): nan},
             {(100, 5): inf, (130, vdim + 63): nan, (256, 2 * vdim + 64): -inf}, {(200, 1): 3.4e38, (255, vdim + 1): -3.4e38}]
    for bad in cases:
        values = v.clone()
        for (at, column), value in bad.items():
            values[at, column] = value
        got, state = run(values)
        touched = torch.zeros_like(got, dtype=torch.bool)
        for (at, column), value in bad.items():
            touched[at:, column] = True
            # The token's own output is its value times q . k, two bfloat16 parts each, beside which the ordinary rest is nothing.
            head = slice(column // vdim * dim, (column // vdim + 1) * dim)
            qt, kt = q[at, head].double(), k[at, head].double()
            want, own = float((qt @ kt * value).float()), float(got[at, column])
            if want == want and abs(want) < inf:
                assert abs(own - want) <= 4 * 2.0 ** -17 * float(qt.norm() * kt.norm()) * abs(value), bad
            else:
                assert own == want or (own != own and want != want), bad
            if not abs(value) < inf:
                assert not torch.isfinite(got[at:, column]).any() and not torch.isfinite(state[column // vdim, :, column % vdim]).any(), bad
        assert torch.equal(got[~touched], clean[~touched]), bad
        untouched = ~torch.isin(torch.arange(heads * vdim, device=cuda_device), torch.tensor([c for _, c in bad], device=cuda_device)).view(heads, 1, vdim)
        assert torch.equal(state[untouched.expand_as(state)], behind[untouched.expand_as(behind)]), bad


# (heads, key channels, value columns, rows, in pieces of 128): us walked and in passes, rotation included.
MEASURED = [((16, 128, 128, [1024, 1024], True), 61.0, 93.7), ((16, 128, 128, [1400, 600], True), 72.7, 93.2), ((16, 128, 128, [700, 400], True), 39.5, 49.0),
            ((16, 128, 128, [1500, 40, 40, 40], True), 74.0, 85.3), ((16, 128, 128, [1500] + [1] * 10, True), 78.8, 96.1),
            ((32, 128, 128, [64] * 16, True), 105.0, 137.8), ((8, 128, 128, [1500, 548], False), 49.6, 58.3), ((8, 128, 128, [1500] + [1] * 10, True), 65.0, 55.4),
            ((5, 100, 132, [300] * 6, True), 26.0, 46.9), ((5, 100, 132, [2048], False), 64.5, 51.7), ((4, 128, 128, [1000], False), 34.5, 24.8),
            ((2, 128, 128, [1500, 548], False), 45.7, 26.4), ((16, 64, 128, [1000], False), 28.7, 41.2), ((16, 64, 128, [1500] + [1] * 10, False), 77.3, 62.4),
            ((4, 64, 64, [2048], False), 43.9, 23.6), ((2, 64, 32, [500], False), 18.2, 19.7)]


@pytest.mark.parametrize("sizes,walked,passes", MEASURED)
def test_steps_take_the_sooner_of_walk_and_passes(cuda_device, sizes, walked, passes):
    from zephyr_b200.kernels import ops
    from zephyr_b200.parts.recurrent import retention_walks

    heads, dim, vdim, lengths, tensor_memory = sizes
    assert ops.retention_in_tensor_memory(len(lengths), sum(lengths), heads, dim, vdim, dim // 2 // 32 * 64) == tensor_memory
    assert retention_walks(lengths, heads, dim, vdim, tensor_memory) == (walked < passes)
