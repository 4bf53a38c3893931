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
