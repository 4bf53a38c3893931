"""The kernels between the products that move whole pieces of four values, against the kernels that take a value at a time: the
same calls with rows that start off a 16-byte boundary, which the latter serve."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


def _apart(x, y, dtype):
    """One step of the result's type (bfloat16 keeps 8 bits: neighbours are up to 2^-7 of their value apart) between float32
    results a few roundings apart: normed and scaled values reach 20, four roundings of 20 * 2^-24 are below 2^-17."""
    step = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -20
    x, y = x.float(), y.float()
    return ((x - y).abs() <= step * torch.maximum(x.abs(), y.abs()) + 2.0 ** -17).all()


class Projected:
    """A fused projection, once with aligned rows and once a value off, with caches for the keys and values of both."""

    def __init__(self, device, dtype, tokens, heads, kv_heads, kd, vd, cached, values=True, seed=0):
        from zephyr_b200.kernels import ops

        g = torch.Generator().manual_seed(seed + tokens + kd)
        dev = lambda t: t.to(device)
        self.width = heads * kd + (kv_heads * (kd + (vd if values else 0)) if cached else 0)
        stride = -(-self.width // 8) * 8
        base = torch.randn(tokens, self.width, generator=g)
        self.rows = [dev(torch.zeros(tokens, stride))[:, :self.width], dev(torch.zeros(tokens, stride + 1))[:, 1:1 + self.width]]
        for r in self.rows:
            r.copy_(base)
        page, blocks = 8, -(-tokens // 8)
        self.table = dev((torch.randperm(blocks, generator=g) + 1).to(torch.int32).view(1, -1))
        self.caches = [dev(torch.zeros(blocks + 1, page * kv_heads * (kd + vd), dtype=dtype)) if cached else None for _ in range(2)]
        self.pos = dev(torch.arange(tokens, dtype=torch.int32))
        self.row = dev(torch.zeros(tokens, dtype=torch.int32))
        self.status = ops.new_status(device)
        self.vector = lambda n: dev(torch.randn(n, generator=g))


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("tokens,heads,kv_heads,kd,vd,rot,form", [
    (700, 16, 4, 128, 128, 128, "norm bias"), (5, 16, 4, 128, 128, 64, "norm"), (601, 9, 1, 20, 24, 12, "unit temp"),
    (640, 30, 3, 100, 60, 0, "bias"), (33, 3, 2, 256, 132, 256, "norm bias temp"), (593, 7, 2, 136, 136, 8, "unit keys"),
    (620, 4, 4, 64, 0, 32, "norm"), (12, 0, 3, 64, 64, 64, "norm"), (611, 11, 2, 64, 64, 64, "queries")])
def test_adjacent_pairs(cuda_device, dtype, tokens, heads, kv_heads, kd, vd, rot, form):
    from zephyr_b200.kernels import ops

    dtype, keys = DTYPES[dtype], "keys" in form
    case = Projected(cuda_device, dtype, tokens, heads, kv_heads, kd, vd, "queries" not in form, values=not keys)
    norm = [case.vector(kd), case.vector(kd)] if "norm" in form else [None, None]
    bias = case.vector(case.width) if "bias" in form else None
    freqs = (1000.0 ** (-torch.arange(rot // 2) / max(rot // 2, 1))).to(cuda_device) if rot else None
    out = [ops.qkv_pairs(rows, heads, kv_heads, kd, vd, bias, *norm, 1e-6, freqs, rot, case.pos, case.row, cache, case.table,
                         case.status, dtype, unit_norm="unit" in form, values_from_keys=keys,
                         q_temp=(0.1, 16) if "temp" in form else None) for rows, cache in zip(case.rows, case.caches)]
    ops.check_status(case.status)
    assert heads == 0 or _apart(*out, dtype)
    assert case.caches[0] is None or (_apart(*case.caches, dtype) and case.caches[0][1:].abs().max() > 0)


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("tokens,heads,kv_heads,kd,vd,rot,form", [
    (700, 16, 4, 128, 128, 128, "per_head bias"), (5, 16, 4, 128, 128, 64, "per_head"), (601, 9, 1, 24, 40, 16, "none unit"),
    (640, 30, 3, 104, 64, 0, "none bias first"), (33, 3, 2, 64, 128, 48, "per_head bias"), (593, 7, 2, 120, 8, 8, "per_head unit first"),
    (611, 11, 2, 64, 64, 64, "none queries")])
def test_halves(cuda_device, dtype, tokens, heads, kv_heads, kd, vd, rot, form):
    from zephyr_b200.kernels import ops

    dtype, mode = DTYPES[dtype], form.split()[0]
    case = Projected(cuda_device, dtype, tokens, heads, kv_heads, kd, vd, "queries" not in form)
    norm = [case.vector(kd), case.vector(kd)] if mode == "per_head" else [None, None]
    bias = case.vector(case.width) if "bias" in form else None
    freqs = (1000.0 ** (-torch.arange(rot // 2) / max(rot // 2, 1))).to(cuda_device) if rot else None
    first = case.vector(tokens * kv_heads * vd).view(tokens, -1) if "first" in form else None
    out = [ops.qkv_halves(rows, heads, kv_heads, kd, vd, mode, *norm, 1e-6, freqs, rot, 1.25, "unit" in form, case.pos, case.row, cache,
                          case.table, case.status, dtype, bias=bias, v_first=first,
                          v_share=torch.tensor([0.3], device=cuda_device) if first is not None else None)
           for rows, cache in zip(case.rows, case.caches)]
    ops.check_status(case.status)
    assert _apart(*out, dtype)
    assert case.caches[0] is None or (_apart(*case.caches, dtype) and case.caches[0][1:].abs().max() > 0)


@pytest.mark.parametrize("group,groups,tokens", [(4, 3, 5), (128, 2, 7), (260, 3, 9), (512, 1, 6), (516, 3, 2), (1024, 2, 33),
                                                 (1028, 1, 3), (2048, 2, 12)])
@pytest.mark.parametrize("gate_first", [False, True])
def test_group_norms(cuda_device, group, groups, tokens, gate_first):
    from zephyr_b200.kernels import ops

    g = torch.Generator().manual_seed(group + tokens)
    width = group * groups
    o, gate, w = torch.randn(tokens, width, generator=g), torch.randn(tokens, width + 4, generator=g), torch.randn(width, generator=g)
    got = ops.gated_group_rms_norm(o.to(cuda_device), gate.to(cuda_device)[:, 4:], w.to(cuda_device), group, 1e-5, gate_first=gate_first)
    act = torch.nn.functional.silu(gate[:, 4:].double())
    x = (o.double() * (act if gate_first else 1.0)).view(tokens, groups, group)
    want = (x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5)).view(tokens, width) * w.double() * (1.0 if gate_first else act)
    # The activation's exponential and five products and sums, each within a few 2^-24 of values up to 20.
    assert (got.cpu().double() - want).abs().max() <= 4e-6 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("group,groups,tokens", [(60, 3, 1000), (64, 1, 2400), (68, 5, 700), (128, 33, 80), (132, 3, 7), (256, 2, 19)])
def test_group_norms_side_by_side(cuda_device, group, groups, tokens):
    """Several groups a warp, one scale for all of them, and gates far out: e^200 is infinite in float32, its inverse zero."""
    from zephyr_b200.kernels import ops

    g = torch.Generator().manual_seed(group + tokens)
    o, gate, w = torch.randn(tokens, group * groups, generator=g), torch.randn(tokens, group * groups, generator=g), torch.randn(group, generator=g)
    gate[0, :4], gate[-1, -4:] = torch.tensor([200.0, -200.0, -88.0, -1e30]), torch.tensor([float("inf"), 1e30, float("-inf"), float("nan")])
    got = ops.gated_group_rms_norm(o.to(cuda_device), gate.to(cuda_device), w.to(cuda_device), group, 1e-5, gate_first=False).cpu().double()
    x = o.double().view(tokens, groups, group)
    want = (x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5)).view(tokens, -1) * w.double().repeat(groups) * torch.nn.functional.silu(gate.double())
    assert torch.equal(got[-1, -4:].isnan(), torch.tensor([False, False, True, True])) and got[-1, -4].isinf()
    got[-1, -4:], want[-1, -4:] = 0.0, 0.0
    # The activation's exponential and five products and sums, each within a few 2^-24 of their own size.
    assert ((got - want).abs() <= 4e-6 * torch.clamp(want.abs(), min=1.0)).all()


@pytest.mark.parametrize("shape", [(1, 4), (3, 5), (129, 516), (1, 2049), (7, 1024)])
def test_sums_and_biases(cuda_device, shape):
    from zephyr_b200.kernels import ops

    g = torch.Generator().manual_seed(shape[1])
    a, b, bias = (torch.randn(n, generator=g).to(cuda_device) for n in (shape, shape, shape[1]))
    for out_dtype in (torch.float32, torch.bfloat16):
        want = (0.75 * a.double() - 1.5 * b.double()).float().to(out_dtype)
        assert _apart(ops.scaled_sum(a, b, 0.75, -1.5, out_dtype=out_dtype), want, out_dtype)
    for dtype in (torch.float32, torch.bfloat16):
        x = a.to(dtype)
        assert torch.equal(ops.add_bias(x.clone(), bias), (x.float() + bias).to(dtype))


@pytest.mark.parametrize("N,K", [(16, 8), (40, 1024), (2048, 2048), (2040, 6152), (4720, 2048), (9472, 256), (9480, 264), (9500, 4104)])
@pytest.mark.parametrize("M", [1, 8, 9, 16, 30, 64])
def test_few_rows_at_the_splits_of_k(cuda_device, N, K, M):
    from zephyr_b200.kernels import ops

    g = torch.Generator(device=cuda_device).manual_seed(N + K + M)
    x = torch.randn(M, K, generator=g, device=cuda_device).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device=cuda_device) / K ** 0.5).to(torch.bfloat16)
    got, want = ops.gemm_small(x, w, out_dtype=torch.float32), x.double() @ w.double().T
    # Exact products of about 1 / sqrt(K), float32 sums of K of them in at most K / 8 + 64 steps: below 2^-24 * sqrt(K) of sums up to 6.
    assert (got.double() - want).abs().max() <= 6 * 2.0 ** -24 * max(16.0, K ** 0.5)
    assert torch.equal(ops.gemm_small(x[M - 1:], w, out_dtype=torch.float32), got[M - 1:])     # a row's sums do not see the others
    if N % 16 == 0:
        gate, up = want.view(M, N // 16, 2, 8).unbind(2)
        hidden = ops.gemm_small(x, w, out_dtype=torch.float32, swiglu=True)
        want = (torch.nn.functional.silu(gate) * up).reshape(M, N // 2)
        assert (hidden.double() - want).abs().max() <= 40 * 2.0 ** -24 * max(16.0, K ** 0.5)


@pytest.mark.parametrize("N,K", [(1528, 2048), (1536, 2056), (2376, 1000), (4720, 4088), (6416, 520), (9488, 40), (9480, 3080), (23680, 1032), (2384, 8200)])
@pytest.mark.parametrize("M", [1, 9, 17])
def test_few_rows_streamed(cuda_device, N, K, M):
    """Around the sizes from which a persistent kernel streams the matrix, also where K ends inside a block or is less than one a
    slice: as exact as the tests above ask, each row alone in the same sums, and the activations behind them."""
    from zephyr_b200.kernels import ops

    g = torch.Generator(device=cuda_device).manual_seed(N + K + M)
    x = torch.randn(M, K + 8, generator=g, device=cuda_device).to(torch.bfloat16)[:, 8:]
    w = (torch.randn(N, K, generator=g, device=cuda_device) / K ** 0.5).to(torch.bfloat16)
    got, want = ops.gemm_small(x, w, out_dtype=torch.float32), x.double() @ w.double().T
    assert (got.double() - want).abs().max() <= 6 * 2.0 ** -24 * max(16.0, K ** 0.5)
    assert torch.equal(ops.gemm_small(x[M - 1:], w, out_dtype=torch.float32), got[M - 1:])
    assert torch.equal(ops.gemm_small(x, w), got.to(torch.bfloat16))
    many = torch.cat([x, x, x, x[:1]] * (1 if M > 9 else 3))[:64]           # through the other kernel where the x of 33 rows and more lies
    assert torch.equal(ops.gemm_small(many, w, out_dtype=torch.float32)[:M], got)
    if N % 16 == 0:
        pair = got.view(M, N // 16, 2, 8)
        gated = ops.gemm_small(x, w, out_dtype=torch.float32, swiglu=True).view(M, N // 16, 8)
        assert (gated - torch.nn.functional.silu(pair[:, :, 0]) * pair[:, :, 1]).abs().max() <= 2.0 ** -21 * max(1.0, float(got.abs().max())) ** 2


@pytest.mark.parametrize("tokens,heads,kv_heads,kd,vd,rot", [(64, 24, 8, 64, 64, 64), (63, 5, 3, 64, 40, 32), (70, 3, 1, 8, 8, 8), (64, 17, 3, 128, 72, 128),
                                                             (700, 31, 5, 88, 128, 40), (2, 1, 1, 56, 64, 24)])
@pytest.mark.parametrize("pairs", [True, False])
def test_heads_side_by_side(cuda_device, tokens, heads, kv_heads, kd, vd, rot, pairs):
    """Heads of a part of a warp, also where a warp holds queries beside keys and keys beside values."""
    from zephyr_b200.kernels import ops

    case = Projected(cuda_device, torch.bfloat16, tokens, heads, kv_heads, kd, vd, True)
    norm, bias = [case.vector(kd), case.vector(kd)], case.vector(case.width)
    freqs = (1000.0 ** (-torch.arange(rot // 2) / (rot // 2))).to(cuda_device)
    out = []
    for rows, cache in zip(case.rows, case.caches):
        where = (freqs, rot), (case.pos, case.row, cache, case.table, case.status, torch.bfloat16)
        out.append(ops.qkv_pairs(rows, heads, kv_heads, kd, vd, bias, *norm, 1e-6, *where[0], *where[1]) if pairs else
                   ops.qkv_halves(rows, heads, kv_heads, kd, vd, "per_head", *norm, 1e-6, *where[0], 1.25, True, *where[1], bias=bias))
    ops.check_status(case.status)
    assert _apart(*out, torch.bfloat16) and _apart(*case.caches, torch.bfloat16) and case.caches[0][1:].abs().max() > 0


@pytest.mark.parametrize("shape", [(1, 4), (3, 5), (129, 516), (12, 2048), (7, 1026)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_a_sum_with_a_bias_is_the_sum_behind_the_bias(cuda_device, shape, out_dtype):
    from zephyr_b200.config.errors import InvalidArgumentError
    from zephyr_b200.kernels import ops

    g = torch.Generator().manual_seed(shape[1])
    a, b, bias = (torch.randn(n, generator=g).to(cuda_device) for n in (shape, shape, shape[1]))
    want = ops.scaled_sum(ops.add_bias(a.clone(), bias), b, 0.75, -1.5, out_dtype=out_dtype)
    assert torch.equal(ops.scaled_sum(a, b, 0.75, -1.5, out_dtype=out_dtype, bias_a=bias), want)
    with pytest.raises(InvalidArgumentError):
        ops.scaled_sum(a, b, 0.75, -1.5, bias_a=bias[:-1])


@pytest.mark.parametrize("N,K,M,streams", [
    (32768, 1024, 8, True), (32768, 768, 8, False), (32768, 256, 1, False), (16384, 512, 8, False), (8192, 1024, 12, False), (4096, 512, 16, False), (2048, 768, 9, False),
    (8192, 1024, 32, False), (4096, 1024, 24, False), (16384, 512, 12, False), (16384, 1024, 8, True), (65536, 512, 5, True), (4096, 1024, 12, True),
    (8192, 512, 12, True), (20480, 256, 12, True), (6144, 1024, 32, True), (32768, 1536, 8, True), (28448, 768, 3, False), (9504, 768, 4, True), (10240, 512, 30, True), (12288, 512, 30, False)])
def test_few_rows_take_the_faster_form(cuda_device, N, K, M, streams):
    """On both sides of the lines between the persistent kernel and the one with bursts (32 rows of the matrix a CTA up to 8 rows): the kernel that was
    the faster one when both were timed, near the exact sums, and the same bits where a row comes alone or with more."""
    from zephyr_b200.kernels import ops

    g = torch.Generator(device=cuda_device).manual_seed(N + K + M)
    x = torch.randn(M, K, generator=g, device=cuda_device).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device=cuda_device) / K ** 0.5).to(torch.bfloat16)
    assert ops.gemm_small_streams(M, N, K) == streams and not ops.gemm_small_streams(33, N, K)
    got = ops.gemm_small(x, w, out_dtype=torch.float32)
    assert (got.double() - x.double() @ w.double().T).abs().max() <= 6 * 2.0 ** -24 * max(16.0, K ** 0.5)
    many = x.repeat(64 // M, 1)
    for rows in (1, 9, 17, 33):
        assert torch.equal(ops.gemm_small(many[:rows], w, out_dtype=torch.float32)[:M], got[:rows])
    if N % 16 == 0:
        pair = got.view(M, N // 16, 2, 8)
        gated = ops.gemm_small(x, w, out_dtype=torch.float32, swiglu=True).view(M, N // 16, 8)
        assert (gated - torch.nn.functional.silu(pair[:, :, 0]) * pair[:, :, 1]).abs().max() <= 2.0 ** -21 * max(1.0, float(got.abs().max())) ** 2


@pytest.mark.parametrize("first,last,step", [(0x00000000, 0x7f800000, 1021), (0x80000000, 0xff800000, 1021), (0xc2ac0000, 0xc2d10000, 1),
                                             (0x80000000, 0x80200000, 1), (0x00000000, 0x00200000, 1), (0xc1000000, 0xc1100000, 1)])
def test_the_activation_over_float32(cuda_device, first, last, step):
    """z / (1 + e^-z) alone, as a convolution of one tap of weight 1, over float32's bit patterns: all magnitudes of either sign, and every value of -86 to
    -104.5 (where 1 + e^-z leaves float32, below which the quotient is a zero), of the smallest, and of some ordinary ones."""
    from zephyr_b200.kernels import ops

    bits = torch.arange(first, last, step, dtype=torch.int64, device=cuda_device)
    z = torch.where(bits >= 2 ** 31, bits - 2 ** 32, bits).to(torch.int32).view(torch.float32)
    channels = 4096
    z = z[:len(z) // channels * channels].view(-1, channels)
    T, i32 = z.shape[0], lambda values: torch.tensor(values, dtype=torch.int32, device=cuda_device)
    got = ops.causal_conv_silu(z, channels, torch.ones(channels, 1, device=cuda_device), torch.zeros(channels, device=cuda_device),
                               torch.zeros(1, 0, device=cuda_device), i32([0]), i32([0]), i32([T]), i32([0] * T), ops.new_status(cuda_device)).double()
    e = torch.exp(-z.double())
    edge = (z.double() + 88.72283905206835).abs() < 1e-4                      # where e^-z is float32's largest
    want = z.double() / (1.0 + torch.where(e > torch.finfo(torch.float32).max, torch.inf, e))
    # The exponential within two steps of 2^-23, its sum and the quotient half a step each; where 1 + e^-z has no more than a few bits as an inverse
    # the correction still has all of them.  Results below float32's normal values: one of their steps.
    assert ((got - want).abs() <= 3.5 * 2.0 ** -23 * want.abs() + 2.0 ** -149)[~edge].all()
    assert (got[edge].abs() <= 1e-36).all()
