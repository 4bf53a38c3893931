"""The float32 product and the float32 attention on the tensor cores, at the edges of their tiles and stages, near the exact sums, and over
values that three bfloat16 parts do not hold."""

import math

import pytest
import torch

from test_kernels_gpu import build_paged_case, ops, rand, ref_attention_row, tiles_for  # noqa: F401  (ops: a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (33, 257, 64), (65, 256, 68), (97, 4096, 132), (700, 4100, 260), (1025, 511, 1024), (200, 19000, 192),
                                   (2049, 3000, 128), (12, 300, 4096)])
def test_product_is_near_the_exact_sums(ops, cuda_device, M, N, K):
    x, w = rand((M, K), torch.float32, cuda_device, 1), rand((N, K), torch.float32, cuda_device, 2)
    got, exact = ops.gemm_nt_simt(x, w).double(), x.double() @ w.double().T
    # A stage of 64 values: four cuts of its sum and a rounding of the total, each at most 2^-23 of the sum so far, and the sum's
    # 2-norm grows with the square root; parts left out 2^-24; the output's rounding 2^-24.
    stages = math.ceil(K / 64)
    assert (got - exact).norm() <= exact.norm() * 2.0 ** -23 * (2 + math.sqrt(stages))
    for row in {0, M // 2, M - 1}:
        assert torch.equal(ops.gemm_nt_simt(x[row:row + 1], w).double(), got[row:row + 1])


def test_values_beyond_the_parts(ops, cuda_device):
    """Infinities, NaN, values that round to infinity in bfloat16 and sums near the smallest: as multiply-adds give them."""
    x, w = rand((70, 256), torch.float32, cuda_device, 3), rand((140, 256), torch.float32, cuda_device, 4)
    x[3, 5], x[4, 6], x[5, 7], w[9, 100] = math.inf, math.nan, 3.4e38, -math.inf
    x[6] *= 1e-36
    got, exact = ops.gemm_nt_simt(x, w), x.double() @ w.double().T
    assert torch.equal(got.isnan(), exact.isnan())
    assert torch.equal(got.isinf(), exact.float().isinf()) and torch.equal(got[got.isinf()], exact.float()[got.isinf()])
    rows = [i for i in range(70) if i not in (3, 4, 5)]
    fine = torch.arange(140, device=cuda_device) != 9
    a, b = got[rows][:, fine].double(), exact[rows][:, fine]
    assert ((a - b).norm(dim=1) <= 256 * 2.0 ** -24 * b.norm(dim=1)).all()


@pytest.mark.parametrize("nh,nkv,hd,window,chunk,q_lens,ctx", [
    (4, 2, 128, 0, 0, [64, 65, 2], [0, 63, 640]), (2, 2, 64, 100, 0, [129, 200], [0, 17]), (40, 1, 60, 0, 96, [7, 30], [90, 0]),
    (64, 1, 128, 0, 0, [5], [127])])
def test_attention_is_near_the_exact_one_and_as_finite_as_the_general_kernel(ops, cuda_device, nh, nkv, hd, window, chunk, q_lens, ctx):
    """Rows and contexts at the edges of a CTA's pairs and of a step's keys; then keys and values that bfloat16 parts do not hold."""
    q, cache, meta, Ks, Vs, qs = build_paged_case(cuda_device, torch.float32, nh, nkv, hd, 16, q_lens, ctx, 100)
    status, wide, tokens = ops.new_status(cuda_device), ops.paged_prefill_tile_tokens(), ops.attention_tile_tokens(nh // nkv)
    common = (meta["row_q_start"], meta["row_q_len"], meta["row_ctx"], nh, nkv, hd, window, 1 / math.sqrt(hd), status)

    def run(held):
        out = torch.empty_like(q)
        ops.paged_attention_f32(q, held, meta["table"], *tiles_for(q_lens, wide, cuda_device, only_multi=True), wide, *common, out, chunk=chunk)
        general = ops.paged_attention(q, held, meta["table"], *tiles_for(q_lens, tokens, cuda_device), tokens, *common, chunk=chunk)
        ops.check_status(status)
        return out, general

    got, general = run(cache)
    cursor = 0
    for r, n in enumerate(q_lens):
        if not chunk:
            exact = ref_attention_row(qs[r].double(), Ks[r].double(), Vs[r].double(), ctx[r], n, window, nh, nkv).view(n, -1)
            # A score: 8 cuts of its sum and one of the small parts', at most 2^-23 of a magnitude of a few; exponential, sum and division
            # two roundings each; 4 cuts a step of keys of the values' sums.
            assert (got[cursor:cursor + n].double().cpu() - exact.cpu()).norm() <= 32 * 2.0 ** -23 * exact.norm()
        cursor += n
    assert (got - general).abs().max() <= 2e-5
    held, at = cache.clone(), ctx[0] + q_lens[0] // 2
    page = meta["table"][0, at // 16]
    held[page, 0, :, at % 16] = 3.4e38                     # a key: its scores reach infinity, of either sign
    held[page, 1, :, at % 16, :4] = 3.4e38                 # and its values
    got, general = run(held)
    assert torch.equal(got.isfinite(), general.isfinite())
    fine = got.isfinite()
    assert ((got - general)[fine].abs() <= 2e-5 * general[fine].abs().clamp(min=1.0)).all()


@pytest.mark.parametrize("nh,nkv,hd,n,ctx", [(2, 1, 128, 5, 150), (8, 2, 60, 40, 130)])
def test_large_values_weigh_what_their_keys_say(ops, cuda_device, nh, nkv, hd, n, ctx):
    """Values that bfloat16 parts do not hold, finite and infinite, at keys of ordinary size, in a row's first step of keys and in later
    ones whose maxima grow: the outputs as numbers, against 64 bits and the general kernel."""
    q, cache, meta, Ks, Vs, qs = build_paged_case(cuda_device, torch.float32, nh, nkv, hd, 16, [n], [ctx], 11)
    status, wide, tokens = ops.new_status(cuda_device), ops.paged_prefill_tile_tokens(), ops.attention_tile_tokens(nh // nkv)
    K, V = Ks[0], Vs[0]
    K *= (torch.arange(ctx + n) / 60.0).view(-1, 1, 1)     # (the largest score of a step grows with its place)
    # In columns 0 .. 5 and hd - 1, each alone in its column: at position 17 (first step), 64 and 100 (second), 128 (third).
    large = {(17, 0): 3.35e38, (17, 1): math.inf, (17, hd - 1): -3.4e38, (64, 2): -math.inf, (100, 3): 3.4e38, (100, 4): math.nan, (128, 5): 3.39e38}
    for (p, column), value in large.items():
        V[p, :, column] = value
    held = cache.clone()
    for p in range(ctx + n):
        where = torch.argsort(ops.kv_row_permutation(p, hd, torch.float32))
        page, off = meta["table"][0, p // 16], p % 16
        held[page, 0, :, off], held[page, 1, :, off] = K[p][:, where].to(cuda_device), V[p][:, where].to(cuda_device)
    common = (meta["row_q_start"], meta["row_q_len"], meta["row_ctx"], nh, nkv, hd, 0, 1 / math.sqrt(hd), status)
    out = torch.empty_like(q)
    ops.paged_attention_f32(q, held, meta["table"], *tiles_for([n], wide, cuda_device), wide, *common, out)
    general = ops.paged_attention(q, held, meta["table"], *tiles_for([n], tokens, cuda_device), tokens, *common)
    ops.check_status(status)
    # Every query sees the large values' keys, so a plain softmax over what it sees is the reference.
    exact = torch.empty(n, nh, hd, dtype=torch.float64)
    for t in range(n):
        for h in range(nh):
            scores = K[:ctx + t + 1, h * nkv // nh].double() @ qs[0][t, h].double() / math.sqrt(hd)
            exact[t, h] = (scores.softmax(0).unsqueeze(1) * V[:ctx + t + 1, h * nkv // nh].double()).sum(0)
    got, general = out.cpu().double().view_as(exact), general.cpu().double().view_as(exact)
    for x in (got, general):
        assert torch.equal(x.isnan(), exact.isnan()) and torch.equal(x.isinf(), exact.isinf())
        assert torch.equal(x[x.isinf()], exact[exact.isinf()])
    # Scores of up to some 30 at errors of 2^-22 of themselves and of the sums behind them move a weight by 2^-17 of itself at most; an ordinary
    # column's values are of about one.
    fine = exact.isfinite()
    assert ((got - exact).abs()[fine] <= 2.0 ** -17 * exact.abs().clamp(min=4.0)[fine]).all()
    assert ((general - exact).abs()[fine] <= 2.0 ** -17 * exact.abs().clamp(min=4.0)[fine]).all()


@pytest.mark.parametrize("M,N,K", [(70, 300, 256), (5, 260, 64), (1500, 515, 68), (33, 40, 516)])
def test_small_values_beside_large_ones(ops, cuda_device, M, N, K):
    """Values below what three bfloat16 parts hold, whose outputs are of any size because the other operand is large: as exact as multiply-adds, and
    every other output keeps its bits."""
    x, w = rand((M, K), torch.float32, cuda_device, 13), rand((N, K), torch.float32, cuda_device, 14)
    plain = ops.gemm_nt_simt(x, w)
    rows = [i for i in (0, M // 2, M - 1)]
    w[1], w[N - 1], w[2], w[N - 2] = w[1] * 2.0 ** 60, w[N - 1] * 1e25, w[2] * 2.0 ** -120, w[N - 2] * 1e-38 * 1e-4
    w[3], w[4] = w[3] * 1e30, w[4] * 1e16                   # (and values and sums beyond the other end)
    x[rows[0]] *= 2.0 ** -125
    x[rows[1]] *= 1e-38
    x[rows[1]] *= 1e-3
    x[rows[2]] = 0.0
    x[rows[2], K - 1] = 1.2345678 * 2.0 ** -120
    got, exact = ops.gemm_nt_simt(x, w), x.double() @ w.double().T
    # K products and sums, each within 2^-24 of what is there, above float32's own smallest steps.
    assert ((got.double() - exact).abs() <= 2.0 ** -24 * K * (x.double().abs() @ w.double().abs().T) + K * 2.0 ** -149).all()
    assert exact[rows[0], 1].abs() > 2.0 ** -80 and exact[rows[1], N - 1].float() != 0
    others, columns = [i for i in range(M) if i not in rows], [j for j in range(N) if j not in (1, 2, 3, 4, N - 1, N - 2)]
    assert torch.equal(got[others][:, columns], plain[others][:, columns])


@pytest.mark.parametrize("key,query,value", [(-122, 60, 0), (0, 0, -122), (-60, 20, 39), (20, 15, 41), (-140, 120, -10), (60, -122, 0)])
def test_attention_holds_values_of_any_size(ops, cuda_device, key, query, value):
    """Keys, queries and values times powers of two, with a scale that takes the scores back: as near the exact averages as ordinary ones."""
    nh, nkv, hd, n, ctx = 4, 2, 68, 70, 100
    q, cache, meta, Ks, Vs, qs = build_paged_case(cuda_device, torch.float32, nh, nkv, hd, 16, [n], [ctx], 21)
    held = cache.clone()
    held[:, 0], held[:, 1], q = held[:, 0] * 2.0 ** (key / 2) * 2.0 ** (key / 2), held[:, 1] * 2.0 ** value, q * 2.0 ** query
    K, V = Ks[0] * 2.0 ** (key / 2) * 2.0 ** (key / 2), Vs[0] * 2.0 ** value
    status, wide, scale = ops.new_status(cuda_device), ops.paged_prefill_tile_tokens(), 2.0 ** -(key + query) / math.sqrt(hd)
    out = torch.empty_like(q)
    ops.paged_attention_f32(q, held, meta["table"], *tiles_for([n], wide, cuda_device), wide, meta["row_q_start"], meta["row_q_len"], meta["row_ctx"],
                            nh, nkv, hd, 0, scale, status, out)
    ops.check_status(status)
    exact = ref_attention_row(qs[0].double(), K.double() * 2.0 ** -key, V.double(), ctx, n, 0, nh, nkv).view(n, -1)
    assert (out.double().cpu() - exact).norm() <= 32 * 2.0 ** -23 * exact.norm()


def test_a_first_product_inside_a_capture(ops, cuda_device, monkeypatch):
    """A graph captured ahead of any other call of the process makes no state that outlives it."""
    x, w = rand((5, 64), torch.float32, cuda_device, 1), rand((70, 64), torch.float32, cuda_device, 2)
    want = ops.gemm_nt_simt(x, w)
    monkeypatch.setattr(ops, "_device_status", {})
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = ops.gemm_nt_simt(x, w)
    assert not ops._device_status
    graph.replay()
    assert torch.equal(got, want)
