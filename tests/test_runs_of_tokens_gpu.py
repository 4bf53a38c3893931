"""Kernels that take runs of tokens instead of single ones, alone, at the edges of their runs and blocks."""

import math

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


@pytest.mark.parametrize("heads,per,dim,vdim", [(4, 2, 128, 64), (6, 3, 64, 20), (3, 1, 40, 36), (2, 2, 16, 130), (40, 8, 128, 64), (2, 1, 8, 9)])
def test_the_state_space_walk(cuda_device, heads, per, dim, vdim):
    """Portions of 33 to 200 tokens and their pieces' edges, from states of their own into them, against the plain
    recurrence; one head's decays are strong (e^-80 a token), one's next to none, both within a piece."""
    from zephyr_b200.kernels import ops

    g = torch.Generator().manual_seed(heads * dim + vdim)
    lengths, slots, groups = [64, 33, 200, 65, 63], [1, 4, 0, 3, 2], heads // per
    T = sum(lengths)
    bf = lambda *shape: torch.randn(*shape, generator=g).to(torch.bfloat16)
    q, k, v, dt = bf(T, groups * dim), bf(T, groups * dim), bf(T, heads * vdim), bf(T, heads)
    a_log, dt_bias, skip = torch.randn(heads, generator=g), torch.randn(heads, generator=g) - 1.0, torch.randn(heads, generator=g)
    a_log[0], a_log[-1] = 3.0, -8.0
    dt[100:103] = 4.0                                       # strong steps in the middle of a piece
    state = torch.randn(5, heads * dim * vdim + 3, generator=g)[:, :heads * dim * vdim]
    dev = lambda t: t.to(cuda_device)
    held = dev(torch.cat([state, torch.zeros(5, 3)], dim=1))[:, :heads * dim * vdim]
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)
    starts = [sum(lengths[:i]) for i in range(len(lengths))]
    status = ops.new_status(cuda_device)
    before = ops.LAUNCH_COUNTS.get("state_walk", 0)
    out = ops.decayed_state_scan("state_space", dev(q), dev(k), dev(v), heads, dim, vdim, held, i32(slots), i32(starts), i32(lengths),
                                 status, dt=dev(dt), dt_bias=dev(dt_bias), a_log=dev(a_log), skip=dev(skip), heads_per_group=per)
    ops.check_status(status)
    assert ops.LAUNCH_COUNTS["state_walk"] == before + 2
    for start, n, slot in zip(starts, lengths, slots):
        S = state[slot].double().view(heads, dim, vdim).clone()
        step = torch.nn.functional.softplus(dt[start:start + n].double() + dt_bias.double())
        decay = torch.exp(-torch.exp(a_log.double()) * step)
        own = torch.arange(heads) // per
        expected = []
        for i in range(n):
            qi, ki = (x[start + i].double().view(groups, dim)[own] for x in (q, k))
            vi = v[start + i].double().view(heads, vdim)
            S = S * decay[i].view(-1, 1, 1) + (ki * step[i].view(-1, 1)).unsqueeze(-1) * vi.unsqueeze(1)
            expected.append(torch.einsum("hdv,hd->hv", S, qi) + skip.double().view(-1, 1) * vi)
        expected = torch.stack(expected).reshape(n, -1)
        # float32 sums of products that are exact, decays good to a few roundings.
        assert (out[start:start + n].cpu().double() - expected).abs().max() <= 3e-6 * max(1.0, float(expected.abs().max()))
        assert (held[slot].cpu().double() - S.reshape(-1)).abs().max() <= 3e-6 * max(1.0, float(S.abs().max()))


@pytest.mark.parametrize("heads,dim,vdim,rot", [(3, 128, 40, 128), (2, 64, 32, 24), (5, 100, 130, 8), (1, 8, 5, 8)])
def test_retention_turns_its_queries_and_keys(cuda_device, heads, dim, vdim, rot):
    """The same portions with q and k turned beforehand and turned on the way into the walk."""
    from zephyr_b200.kernels import ops

    g = torch.Generator().manual_seed(dim + vdim)
    lengths, slots = [64, 100, 7, 130], [1, 0, 3, 2]
    T, hd = sum(lengths), heads * dim
    dev = lambda t: t.to(cuda_device)
    projected = dev(torch.randn(T, (2 * hd + heads * vdim + 3) // 4 * 4, generator=g))
    freqs = dev(10000.0 ** (-torch.arange(rot // 2) / (rot // 2)))
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)
    positions = i32([p + 500 * r for r, n in enumerate(lengths) for p in range(n)])
    decay = dev(1.0 - 2.0 ** -(1.0 + 3.0 * torch.arange(heads)))
    starts = [sum(lengths[:i]) for i in range(len(lengths))]
    status, got = ops.new_status(cuda_device), []
    turned = ops.rotate_qk(projected, heads, dim, freqs, rot, dim ** -0.5, positions)
    for q, k, turn in ((turned[:, :hd], turned[:, hd:], {}),
                       (projected[:, :hd], projected[:, hd:2 * hd], dict(freqs=freqs, rot_dims=rot, k_scale=dim ** -0.5, positions=positions))):
        assert not turn or ops.retention_turns(q, k, dim, rot)
        state = torch.ones(4, hd * vdim, device=cuda_device)
        got.append((ops.retention(q, k, projected[:, 2 * hd:2 * hd + heads * vdim], decay, heads, dim, vdim, state, i32(slots), i32(starts),
                                  i32(lengths), status, **turn), state))
    ops.check_status(status)
    for x, y in zip(*got):       # the same float32 rotation, at most a rounding apart ahead of the split
        assert (x - y).abs().max() <= 4e-6 * max(1.0, float(x.abs().max()))


@pytest.mark.parametrize("kind", ["delta", "state_space", "retention"])
def test_rows_whose_tokens_lie_in_another_order(cuda_device, kind):
    """Rows may name any stretch of the stream: listed backwards or shuffled they get the bits they get in the stream's
    order.  (Lengths at which numbers counted from a row's first token would meet: 40 and 40, the second row first.)"""
    from zephyr_b200.kernels import ops

    heads, per, dim, vdim = 4, 2 if kind != "retention" else 1, 64, 48
    lengths = [40, 40, 200, 64, 33, 97]
    starts, T, groups = [sum(lengths[:i]) for i in range(len(lengths))], sum(lengths), heads // per
    g = torch.Generator().manual_seed(9)
    dtype = torch.bfloat16 if kind == "state_space" else torch.float32
    q, k, v, b, a = (torch.randn(T, n, generator=g).to(cuda_device) for n in (groups * dim, groups * dim, heads * vdim, heads, heads))
    q, k, v, dt = (t.to(dtype) for t in (q, k, v, a))
    constants = [(torch.rand(heads, generator=g) - 0.5).to(cuda_device) for _ in range(3)]
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)
    status = ops.new_status(cuda_device)

    def run(order):
        state = torch.zeros(len(lengths), heads * dim * vdim, device=cuda_device)
        rows = (state, i32(order), i32([starts[r] for r in order]), i32([lengths[r] for r in order]), status)
        if kind == "delta":
            out = ops.delta_rule(q, k, v, b, a, constants[0], constants[1], heads, groups, dim, vdim, *rows, q_scale=dim ** -0.5)
        elif kind == "retention":
            out = ops.retention(q, k, v, constants[0].abs() + 0.4, heads, dim, vdim, *rows)
        else:
            out = ops.decayed_state_scan("state_space", q, k, v, heads, dim, vdim, *rows, dt=dt, dt_bias=constants[0],
                                         a_log=constants[1], skip=constants[2], heads_per_group=per)
        ops.check_status(status)
        return out, state

    expected = run(list(range(len(lengths))))
    for order in ([1, 0, 2, 3, 4, 5], [5, 4, 3, 2, 1, 0], [2, 5, 0, 4, 1, 3]):
        for x, y in zip(run(order), expected):
            assert torch.equal(x, y), order


def _delta_in_float64(q, k, v, b, a, a_log, dt_bias, heads, groups, dim, vdim, state):
    """The plain rule, from the state [heads, vdim, dim] on: outputs [T, heads, vdim] and the state behind them."""
    T, own = len(v), torch.arange(heads) // (heads // groups)
    q, k, v, b, a, a_log, dt_bias, S = (t.cpu().double() for t in (q, k, v, b, a, a_log, dt_bias, state))
    unit = lambda x: (x.view(T, groups, dim) / torch.sqrt((x.view(T, groups, dim) ** 2).sum(-1, keepdim=True) + 1e-6))[:, own]
    q, k, v, S = unit(q) * dim ** -0.5, unit(k), v.view(T, heads, vdim), S.view(heads, vdim, dim).clone()
    beta, decay = torch.sigmoid(b), torch.exp(-torch.exp(a_log) * torch.nn.functional.softplus(a + dt_bias))
    out = torch.zeros(T, heads, vdim, dtype=torch.float64)
    for t in range(T):
        S = S * decay[t].view(-1, 1, 1)
        u = beta[t].view(-1, 1) * (v[t] - torch.einsum("hvd,hd->hv", S, k[t]))
        S = S + u.unsqueeze(-1) * k[t].unsqueeze(1)
        out[t] = torch.einsum("hvd,hd->hv", S, q[t])
    return out, S


@pytest.mark.parametrize("dim,vdim", [(128, 64), (48, 20)])
def test_the_delta_rule_in_blocks_keeps_float32(cuda_device, dim, vdim):
    """With rates and steps as such models start them, blocks are as close to 64 bits as the token-by-token form, which portions
    of 15 tokens take: sums in another order, of the same precision."""
    from zephyr_b200.kernels import ops

    heads, groups, T = 4, 2, 512
    g = torch.Generator().manual_seed(dim)
    q, k, v, b, a = (torch.randn(T, n, generator=g) for n in (groups * dim, groups * dim, heads * vdim, heads, heads))
    step = torch.exp(torch.rand(heads, generator=g) * math.log(100.0) - math.log(1000.0))
    a_log, dt_bias = torch.log(1.0 + 15.0 * torch.rand(heads, generator=g)), step + torch.log(-torch.expm1(-step))
    ba = torch.cat([b, a], dim=1).to(cuda_device)
    dev = lambda t: t.to(cuda_device)
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)
    status = ops.new_status(cuda_device)
    expected, last = _delta_in_float64(q, k, v, b, a, a_log, dt_bias, heads, groups, dim, vdim, torch.zeros(heads, vdim, dim))

    def error(cuts):
        state, out, at = torch.zeros(1, heads * dim * vdim, device=cuda_device), [], 0
        for n in cuts:
            part = slice(at, at + n)
            out.append(ops.delta_rule(dev(q[part]), dev(k[part]), dev(v[part]), ba[part, :heads], ba[part, heads:], dev(a_log), dev(dt_bias),
                                      heads, groups, dim, vdim, state, i32([0]), i32([0]), i32([n]), status, q_scale=dim ** -0.5))
            at += n
        ops.check_status(status)
        got = torch.cat(out).cpu().double().view_as(expected)
        return float((got - expected).norm() / expected.norm()), float((state.cpu().double().view_as(last) - last).norm() / last.norm())

    # (measured over such inputs: 0.7 to 0.9 of the token-by-token form's error; operands of two TF32 values: 1.5 to 1.9)
    for blocks, tokens in zip(error([T]), error([15] * (T // 15) + [T % 15])):
        assert blocks <= 1.2 * tokens


@pytest.mark.parametrize("rate", [50.0, 300.0, 3000.0, math.inf])
def test_the_delta_rule_behind_a_token_that_forgets(cuda_device, rate):
    """Tokens with logarithms of their decays of -rate in front of tokens that forget next to nothing: what the latter give
    and the state behind them are as good as without the former, and a decay of exactly zero is a zero."""
    from zephyr_b200.kernels import ops

    heads, groups, dim, vdim, T = 2, 1, 64, 32, 96
    g = torch.Generator().manual_seed(6)
    q, k, v, b = (torch.randn(T, n, generator=g) for n in (groups * dim, groups * dim, heads * vdim, heads))
    # A step of softplus(a) at a rate of e^3: -8 is next to no decay, a large one e^(-20 a).
    a, a_log = torch.full((T, heads), -8.0), torch.full((heads,), 3.0)
    strong = [0, 1, 17, 32, 33, 50, 80]
    a[strong] = min(rate / math.exp(3.0), 3e38)
    b += 2.0
    ba = torch.cat([b, a], dim=1).to(cuda_device)
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)
    state, status = torch.ones(1, heads * dim * vdim, device=cuda_device), ops.new_status(cuda_device)
    expected, last = _delta_in_float64(q, k, v, b, a, a_log, torch.zeros(heads), heads, groups, dim, vdim, state)
    out = ops.delta_rule(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device), ba[:, :heads], ba[:, heads:], a_log.to(cuda_device),
                         torch.zeros(heads, device=cuda_device), heads, groups, dim, vdim, state, i32([0]), i32([0]), i32([T]), status,
                         q_scale=dim ** -0.5)
    ops.check_status(status)
    # Sums over 64 channels and up to 30 tokens of memory in float32: some tens of roundings of 2^-24 of the largest value.
    behind = torch.tensor([t for t in range(T) if t not in strong])
    got, want = out.cpu().double().view(T, heads, vdim)[behind], expected[behind]
    assert (got - want).abs().max() <= 2e-6 * float(want.abs().max())
    assert (state.cpu().double().view_as(last) - last).abs().max() <= 2e-6 * float(last.abs().max())


@pytest.mark.parametrize("kind", ["delta", "state_space", "retention"])
def test_a_value_that_is_not_finite_stays_with_later_tokens(cuda_device, kind):
    """An infinity or a NaN in one value of a token: all tokens before it, and all other columns, keep their bits."""
    from zephyr_b200.kernels import ops

    heads, per, dim, vdim, T = 4, 2 if kind != "retention" else 1, 64, 48, 150
    groups, g = heads // per, torch.Generator().manual_seed(4)
    dtype = torch.bfloat16 if kind == "state_space" else torch.float32
    q, k, v, b, a = (torch.randn(T, n, generator=g).to(cuda_device) for n in (groups * dim, groups * dim, heads * vdim, heads, heads))
    q, k, v, dt = (t.to(dtype) for t in (q, k, v, a))
    constants = [(torch.rand(heads, generator=g) - 0.5).to(cuda_device) for _ in range(3)]
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)
    status = ops.new_status(cuda_device)

    def run(values):
        rows = (torch.zeros(1, heads * dim * vdim, device=cuda_device), i32([0]), i32([0]), i32([T]), status)
        if kind == "delta":
            return ops.delta_rule(q, k, values, b, a, constants[0], constants[1], heads, groups, dim, vdim, *rows, q_scale=dim ** -0.5)
        if kind == "retention":
            return ops.retention(q, k, values, constants[0].abs() + 0.4, heads, dim, vdim, *rows)
        return ops.decayed_state_scan("state_space", q, k, values, heads, dim, vdim, *rows, dt=dt, dt_bias=constants[0], a_log=constants[1],
                                      skip=constants[2], heads_per_group=per)

    clean = run(v)
    for at, bad in ((0, math.nan), (7, math.inf), (15, -math.inf), (16, math.inf), (37, math.nan), (63, math.inf), (70, math.inf), (149, math.nan)):
        values, column = v.clone(), (2 * at + 5) % (heads * vdim)
        values[at, column] = bad
        got, others = run(values), torch.arange(heads * vdim, device=cuda_device) != column
        ops.check_status(status)
        assert torch.equal(got[:at], clean[:at]), at
        assert torch.equal(got[:, others], clean[:, others]), at
        assert not torch.isfinite(got[at:, column]).any(), at


@pytest.mark.parametrize("dim,vdim", [(128, 64), (64, 40)])
def test_the_state_space_walk_keeps_float32(cuda_device, dim, vdim):
    """With rates and steps as such models start them, the walk over pieces is as close to 64 bits as the scan over tokens."""
    from zephyr_b200.kernels import ops

    heads, per, T = 8, 4, 700
    groups, g = heads // per, torch.Generator().manual_seed(dim)
    bf = lambda *shape: torch.randn(*shape, generator=g).to(torch.bfloat16)
    q, k, v, dt = bf(T, groups * dim), bf(T, groups * dim), bf(T, heads * vdim), bf(T, heads)
    step = torch.exp(torch.rand(heads, generator=g) * math.log(100.0) - math.log(1000.0))
    a_log, dt_bias = torch.log(1.0 + 15.0 * torch.rand(heads, generator=g)), step + torch.log(-torch.expm1(-step))
    skip = torch.randn(heads, generator=g)
    dev = lambda t: t.to(cuda_device)
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)
    status, own = ops.new_status(cuda_device), torch.arange(heads) // per
    taken = torch.nn.functional.softplus(dt.double() + dt_bias.double())
    decay = torch.exp(-torch.exp(a_log.double()) * taken)
    S, expected = torch.zeros(heads, dim, vdim, dtype=torch.float64), torch.zeros(T, heads, vdim, dtype=torch.float64)
    for t in range(T):
        values = v[t].double().view(heads, vdim)
        S = S * decay[t].view(-1, 1, 1) + (k[t].double().view(groups, dim)[own] * taken[t].view(-1, 1)).unsqueeze(-1) * values.unsqueeze(1)
        expected[t] = torch.einsum("hdv,hd->hv", S, q[t].double().view(groups, dim)[own]) + skip.double().view(-1, 1) * values

    def error(segment):
        state = torch.zeros(1, heads * dim * vdim, device=cuda_device)
        out = ops.decayed_state_scan("state_space", dev(q), dev(k), dev(v), heads, dim, vdim, state, i32([0]), i32([0]), i32([T]), status,
                                     dt=dev(dt), dt_bias=dev(dt_bias), a_log=dev(a_log), skip=dev(skip), heads_per_group=per, segment=segment)
        ops.check_status(status)
        return (float((out.cpu().double().view_as(expected) - expected).norm() / expected.norm()),
                float((state.cpu().double().view_as(S) - S).norm() / S.norm()))

    for walk, scan in zip(error(None), error(0)):
        assert walk <= 1.15 * scan, (walk, scan)


@pytest.mark.parametrize("kind", ["delta", "state_space"])
def test_what_a_row_gets_hangs_on_that_row_alone(cuda_device, kind):
    """Portions of many sizes in one step, and each in a step of its own: the same bits, whether the host knows the rows'
    sizes or not."""
    from zephyr_b200.kernels import ops

    heads, per, dim, vdim = 4, 2, 64, 48
    lengths = [1, 100, 1, 1, 15, 16, 1, 300, 1, 1, 63, 64, 1, 1, 31, 32, 2, 1, 1, 1]
    starts, T, groups = [sum(lengths[:i]) for i in range(len(lengths))], sum(lengths), heads // per
    g = torch.Generator().manual_seed(3)
    dtype = torch.bfloat16 if kind == "state_space" else torch.float32
    q, k, v, b, a = (torch.randn(T, n, generator=g).to(cuda_device) for n in (groups * dim, groups * dim, heads * vdim, heads, heads))
    q, k, v, dt = (t.to(dtype) for t in (q, k, v, a))
    constants = [(torch.rand(heads, generator=g) - 0.5).to(cuda_device) for _ in range(3)]
    before = torch.randn(len(lengths), heads * dim * vdim, generator=g).to(cuda_device)
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)
    status = ops.new_status(cuda_device)

    def run(rows, **more):
        first, end = starts[rows[0]], starts[rows[-1]] + lengths[rows[-1]]
        part, state = slice(first, end), before.clone()
        where = (state, i32(rows), i32([starts[r] - first for r in rows]), i32([lengths[r] for r in rows]), status)
        if kind == "delta":
            out = ops.delta_rule(q[part], k[part], v[part], b[part], a[part], constants[0], constants[1], heads, groups, dim, vdim, *where,
                                 q_scale=dim ** -0.5, **more)
        else:
            out = ops.decayed_state_scan("state_space", q[part], k[part], v[part], heads, dim, vdim, *where, dt=dt[part],
                                         dt_bias=constants[0], a_log=constants[1], skip=constants[2], heads_per_group=per, **more)
        ops.check_status(status)
        return out, state

    together = [run(list(range(len(lengths))), **more) for more in ({}, {"row_tokens": lengths})]
    for out, state in together[1:]:
        assert torch.equal(out, together[0][0]) and torch.equal(state, together[0][1])
    for r, (start, n) in enumerate(zip(starts, lengths)):
        out, state = run([r])
        assert torch.equal(together[0][0][start:start + n], out), n
        assert torch.equal(together[0][1][r], state[r]), n


@pytest.mark.parametrize("heads,dim,vdim", [(2, 64, 32), (5, 100, 130), (1, 8, 8)])
def test_retention_walked_and_in_passes(cuda_device, heads, dim, vdim):
    """The two forms that a layer chooses from by its state's size: the same rule, each operand two bfloat16 values."""
    from zephyr_b200.kernels import ops

    g = torch.Generator().manual_seed(dim)
    lengths, T = [64, 100, 7, 130], 301
    q, k, v = (torch.randn(T, heads * n, generator=g).to(cuda_device) for n in (dim, dim, vdim))
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)
    rows = (i32([1, 0, 3, 2]), i32([0, 64, 164, 171]), i32(lengths), ops.new_status(cuda_device))
    decay, got = torch.full((heads,), 0.98, device=cuda_device), []
    for walk in (True, False):
        before, state = ops.LAUNCH_COUNTS.get("state_walk", 0), torch.ones(4, heads * dim * vdim, device=cuda_device)
        got.append((ops.retention(q, k, v, decay, heads, dim, vdim, state, *rows, walk=walk), state))
        assert ops.LAUNCH_COUNTS.get("state_walk", 0) - before == (2 if walk else 0)
    ops.check_status(rows[-1])
    # An operand is off by 2^-17 of itself at most in either form; sums of up to 130 products, of alternating signs.
    for x, y in zip(*got):
        assert (x - y).norm() <= 2.0 ** -15 * y.norm()
