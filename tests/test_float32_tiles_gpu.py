"""The 32-bit kernels alone: the product at the edges of its tiles and of its slices of k (on the tensor cores where rows start on 16-byte
boundaries, in register tiles elsewhere), and the attention over rows with several tokens against the general kernel and a plain
float64 attention."""

import math

import pytest
import torch

from test_kernels_gpu import build_paged_case, ops, rand, ref_attention_row, tiles_for  # noqa: F401  (ops: a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 32, 4), (31, 33, 64), (33, 100, 60), (64, 128, 16), (700, 1024, 132), (640, 1000, 1028),
                                   (1281, 515, 68)])
def test_product_at_tile_edges(ops, cuda_device, M, N, K):
    x, w = rand((M, K), torch.float32, cuda_device, 1), rand((N, K), torch.float32, cuda_device, 2)
    got = ops.gemm_nt_simt(x, w)
    # A sum of K products: every partial sum is rounded, at most K of them of magnitude up to sqrt(K) times a few.
    assert (got.double() - x.double() @ w.double().T).abs().max() <= 6 * 2.0 ** -24 * math.sqrt(K) * math.sqrt(K)
    # A row's sums are the same on either tile size and in a batch of any size.
    assert torch.equal(ops.gemm_nt_simt(x[M - 1:], w), got[M - 1:])
    # Rows that lie apart, in and out; what lies between them stays.
    wide = torch.full((M, N + 3), 7.0, device=cuda_device)
    ops.gemm_nt_simt(rand((M, K), torch.float32, cuda_device, 1).repeat(1, 2)[:, :K], w, out=wide[:, :N])
    assert torch.equal(wide[:, :N], got) and bool((wide[:, N:] == 7.0).all())


@pytest.mark.parametrize("nh,nkv,hd,page,window,chunk,softcap,sink", [
    (4, 2, 16, 4, 0, 0, 0.0, False), (16, 8, 128, 16, 0, 0, 0.0, False), (6, 2, 64, 8, 24, 0, 0.0, True),
    (9, 1, 68, 16, 0, 40, 0.0, False), (40, 1, 112, 16, 0, 0, 5.0, True), (3, 3, 100, 32, 70, 0, 0.0, False)])
def test_attention_against_the_general_kernel(ops, cuda_device, nh, nkv, hd, page, window, chunk, softcap, sink):
    q_lens, ctx = [1, 37, 2, 150, 64, 129], [130, 0, 63, 3, 64, 200]
    q, cache, meta, Ks, Vs, qs = build_paged_case(cuda_device, torch.float32, nh, nkv, hd, page, q_lens, ctx, 100)
    sinks = rand((nh,), torch.float32, cuda_device, 5) if sink else None
    status = ops.new_status(cuda_device)
    common = (meta["row_q_start"], meta["row_q_len"], meta["row_ctx"], nh, nkv, hd, window, 1 / math.sqrt(hd), status)
    masks = dict(chunk=chunk, sinks=sinks, softcap=softcap)
    tokens = ops.attention_tile_tokens(nh // nkv)
    general = ops.paged_attention(q, cache, meta["table"], *tiles_for(q_lens, tokens, cuda_device), tokens, *common, **masks)
    wide = ops.paged_prefill_tile_tokens()
    out = torch.full_like(q, 7.0)
    ops.paged_attention_f32(q, cache, meta["table"], *tiles_for(q_lens, wide, cuda_device, only_multi=True), wide, *common, out, **masks)
    ops.check_status(status)
    assert bool((out[:1] == 7.0).all())                   # the single token is another kernel's
    # Two float32 softmax averages of values around one: a few roundings of the scores' products and of the sums.
    assert (out[1:] - general[1:]).abs().max() <= 2e-5
    if not (chunk or softcap or sink):
        got, cursor = out.double().cpu().view(-1, nh, hd), 0
        for r, n in enumerate(q_lens):
            expected = ref_attention_row(qs[r].double(), Ks[r].double(), Vs[r].double(), ctx[r], n, window, nh, nkv)
            assert n == 1 or (got[cursor:cursor + n] - expected).abs().max() <= 4e-5
            cursor += n


def test_attention_refuses_what_it_does_not_take(ops):
    assert ops.paged_attention_f32_supported(64, 1, 128, torch.float32)
    for nh, nkv, hd, dtype in ((65, 1, 64, torch.float32), (4, 2, 132, torch.float32), (4, 2, 30, torch.float32), (4, 2, 64, torch.bfloat16)):
        assert not ops.paged_attention_f32_supported(nh, nkv, hd, dtype)


@pytest.mark.parametrize("nh,nkv,hd,window,chunk", [(4, 2, 64, 0, 0), (3, 1, 128, 40, 0), (2, 2, 20, 0, 50)])
def test_values_that_are_not_finite_stay_with_the_tokens_that_see_them(ops, cuda_device, nh, nkv, hd, window, chunk):
    """An infinity and a NaN among the values of one position: every query that does not see it keeps its bits."""
    n, ctx, page = 150, 30, 16
    q, cache, meta, *_ = build_paged_case(cuda_device, torch.float32, nh, nkv, hd, page, [n], [ctx], 7)
    status, wide = ops.new_status(cuda_device), ops.paged_prefill_tile_tokens()

    def run(held):
        out = torch.empty_like(q)
        ops.paged_attention_f32(q, held, meta["table"], *tiles_for([n], wide, cuda_device), wide, meta["row_q_start"], meta["row_q_len"],
                                meta["row_ctx"], nh, nkv, hd, window, 1 / math.sqrt(hd), status, out, chunk=chunk)
        ops.check_status(status)
        return out

    clean = run(cache)
    for at in (17, 63, 64, 100, ctx + n - 1):
        held = cache.clone()
        held[meta["table"][0, at // page], 1, :, at % page, 0::2] = math.inf
        held[meta["table"][0, at // page], 1, :, at % page, 1::2] = math.nan
        got, position = run(held), torch.arange(ctx, ctx + n, device=cuda_device)
        sees = position >= at
        if window:
            sees &= position - at < window
        if chunk:
            sees &= position // chunk == at // chunk
        assert torch.equal(got[~sees], clean[~sees]), at
        assert not torch.isfinite(got[sees]).any()


@pytest.mark.parametrize("M,N,K,apart", [(70, 311, 200, 3), (70, 311, 203, 0), (5, 33, 64, 2), (1300, 515, 68, 1), (33, 40, 16, 4)])
def test_a_rows_sums_do_not_depend_on_the_batch(ops, cuda_device, M, N, K, apart):
    """Rows that lie apart by any stride, alone and in a batch, and the outputs of one row of w alone: the same bits."""
    wide, w = rand((M, K + apart), torch.float32, cuda_device, 3), rand((N, K + apart), torch.float32, cuda_device, 4)
    x, w = wide[:, :K], w[:, :K]
    got = ops.gemm_nt_simt(x, w)
    assert (got.double() - x.double() @ w.double().T).abs().max() <= 6 * 2.0 ** -24 * K
    for i in (0, 1, M // 2, M - 1):
        assert torch.equal(ops.gemm_nt_simt(x[i:i + 1], w), got[i:i + 1])
    for j in (0, N - 1):
        assert torch.equal(ops.gemm_nt_simt(x, w[j:j + 1]), got[:, j:j + 1])


def test_float32_logits_do_not_depend_on_what_shares_the_step(model_folders, cuda_device):
    """Prompts of 40, 17 and 3 tokens and single tokens behind some of them, in steps of their own and in one step with
    many others: the same bits."""
    from replay_util import random_tokens
    from tiny_configs import TINY
    from zephyr_b200.config import load_model_spec
    from zephyr_b200.engine import ModelRunner, StepEntry
    from zephyr_b200.parts import Model
    from zephyr_b200.weights import Checkpoint

    folder = model_folders("D", "float32")
    model = Model.load(load_model_spec(folder), Checkpoint(folder), torch.float32, cuda_device)
    lengths = [40, 1, 17, 3] + [1] * 12
    tokens = [random_tokens(TINY["D"]["config"]["vocab_size"], 2 * n, seed=i) for i, n in enumerate(lengths)]

    def logits(groups):
        runner, out = ModelRunner(model, TINY["D"]["page_size"], 64, len(lengths), use_cuda_graphs=False), {}
        for r in range(len(lengths)):
            assert runner.add_request(r)
        for half in (0, 1):
            for group in groups:
                got = runner.step([StepEntry(r, tokens[r][half * lengths[r]:(half + 1) * lengths[r]], (lengths[r] - 1,)) for r in group])
                out.update({(r, half): got[i].clone() for i, r in enumerate(group)})
        runner.check()
        return out

    alone, together = logits([[r] for r in range(len(lengths))]), logits([list(range(len(lengths)))])
    for key in alone:
        assert torch.equal(alone[key], together[key]), key


@pytest.mark.parametrize("m,n,k", [
    (700, 1000, 60), (1500, 1023, 36), (300, 1030, 132), (129, 4100, 68), (64, 4096, 64), (33, 6145, 20), (200, 1024, 100), (2048, 4097, 16),
    (8, 70001, 12), (1, 5, 4),
    (2100000, 5, 4)])
def test_products_in_every_tile(ops, cuda_device, m, n, k):
    """Whatever tile the sizes choose: near the exact product, and a row's sums the same to the bit as on its own."""
    x, w = rand((m, k), torch.float32, cuda_device, 70), rand((n, k), torch.float32, cuda_device, 71)
    got, exact = ops.gemm_nt_simt(x, w), x.double() @ w.double().T
    assert (got.double() - exact).abs().max() <= k * 2.0 ** -24 * float((x.abs().double() @ w.abs().double().T).max())
    for row in {0, m // 2, m - 1}:
        assert torch.equal(got[row:row + 1], ops.gemm_nt_simt(x[row:row + 1], w))
