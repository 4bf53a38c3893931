"""The prompt kernel on tcgen05 in both forms of a CTA (two heads; one head whose tiles of keys two slots take by turns), and over
rows that are keys and values at once, at the edges of its tiles, against a plain float64 attention.  The cache holds NaN wherever
no request's row lies."""

import dataclasses
import math

import pytest
import torch

from test_kernels_gpu import build_paged_case, make_tables, ops, rand, tiles_for  # noqa: F401  (ops: a fixture)

pytestmark = pytest.mark.gpu

# Probabilities and the result are rounded to bfloat16: 2^-9 of a value of up to four each, and what the weights' roundings
# add up to over a row stays below the larger of them.
BOUND = 3.2e-2


def plain(q, K, V, ctx, scale, sinks=None, softcap=0.0, window=0):
    """q [T, heads, d] behind ``ctx`` positions of K [ctx + T, groups, d], V [ctx + T, groups, dv]."""
    T, nh = q.shape[:2]
    i, j = torch.arange(ctx, ctx + T)[:, None], torch.arange(ctx + T)[None, :]
    seen = (j <= i) & ((i - j < window) if window else (j <= i))
    out = []
    for h in range(nh):
        g = h // (nh // K.shape[1])
        s = q[:, h].double() @ K[:, g].double().T * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(~seen, -math.inf)
        if sinks is not None:
            s = torch.cat([s, sinks[h].double().expand(T, 1)], dim=1)
        out.append(torch.softmax(s, -1)[:, :ctx + T] @ V[:, g].double())
    return torch.stack(out, 1)


def in_order_of_keys(tiles, q_lens, ctx):
    """The tiles as the engine lists them: by the number of keys they see, fewest first."""
    rows, q0s = tiles
    keys = torch.tensor([ctx[r] + min(q0 + 128, q_lens[r]) for r, q0 in zip(rows.tolist(), q0s.tolist())])
    order = torch.argsort(keys, stable=True).to(rows.device)
    return rows[order], q0s[order]


@pytest.mark.parametrize("nh,nkv,q_lens,ctx,page,sink,softcap,window", [
    (2, 1, [1], [0], 16, False, 0.0, 0),                                  # one tile: the second slot has none
    (2, 1, [128], [128], 16, True, 0.0, 0), (2, 1, [129], [127], 8, False, 0.0, 0),
    (3, 1, [257, 3], [0, 383], 16, True, 0.0, 0),                         # heads without a partner
    (6, 2, [300], [84], 32, False, 25.0, 0), (1, 1, [140], [1000], 16, False, 0.0, 150),
    (32, 8, [640, 100], [0, 300], 16, True, 0.0, 0),                      # more CTAs than SMs, long rows: heads singly
    (32, 8, [130, 1, 127, 128, 90, 64], [0, 511, 129, 128, 64, 1], 16, False, 0.0, 0),      # many rows: pairs
    (32, 8, [500, 40, 40], [100, 0, 700], 128, True, 30.0, 0), (40, 4, [200, 200, 7], [0, 60, 400], 16, False, 0.0, 130)])
def test_two_slots(ops, cuda_device, nh, nkv, q_lens, ctx, page, sink, softcap, window):
    hd = 128
    q, cache, meta, Ks, Vs, qs = build_paged_case(cuda_device, torch.bfloat16, nh, nkv, hd, page, q_lens, ctx, 400)
    sinks = rand((nh,), torch.float32, cuda_device, 6) if sink else None
    status, before = ops.new_status(cuda_device), ops.LAUNCH_COUNTS.get("paged_prefill_tc", 0)
    tiles = in_order_of_keys(tiles_for(q_lens, ops.paged_prefill_tile_tokens(), cuda_device), q_lens, ctx)
    got = ops.paged_prefill(q, cache, meta["table"], *tiles, meta["row_q_start"], meta["row_q_len"], meta["row_ctx"], nh, nkv, hd,
                            window, 1 / math.sqrt(hd), status, torch.full_like(q, float("nan")), sinks=sinks, softcap=softcap)
    ops.check_status(status)
    assert ops.LAUNCH_COUNTS["paged_prefill_tc"] == before + 1
    at = 0
    for r, n in enumerate(q_lens):
        expected = plain(qs[r], Ks[r], Vs[r], ctx[r], 1 / math.sqrt(hd), sinks.cpu() if sink else None, softcap, window)
        assert (got[at:at + n].double().cpu().view(n, nh, hd) - expected).abs().max() <= BOUND
        at += n


def test_scores_that_grow_from_tile_to_tile(ops, cuda_device):
    """Every tile of keys raises a row's largest score by more than the shift may lag, in both forms of a CTA."""
    for nh, nkv, q_lens in ((2, 1, [513]), (32, 8, [513])):
        hd, ctx = 128, [0]
        q, cache, meta, Ks, Vs, qs = build_paged_case(cuda_device, torch.bfloat16, nh, nkv, hd, 16, q_lens, ctx, 410)
        q = (q.float().abs() * 0 + 1.0).to(q.dtype)
        steps = (torch.arange(q_lens[0]) // 100).float()                   # score 0.088 * 128 * 2 * step: 22 a step
        for p in range(q_lens[0]):
            page = int(meta["table"][0, p // 16])
            cache[page, 0, :, p % 16] = 2.0 * steps[p]
            Ks[0][p] = 2.0 * steps[p]
        status = ops.new_status(cuda_device)
        tiles = in_order_of_keys(tiles_for(q_lens, ops.paged_prefill_tile_tokens(), cuda_device), q_lens, ctx)
        got = ops.paged_prefill(q, cache, meta["table"], *tiles, meta["row_q_start"], meta["row_q_len"], meta["row_ctx"], nh, nkv, hd,
                                0, 1 / math.sqrt(hd), status, torch.empty_like(q))
        ops.check_status(status)
        expected = plain(torch.ones_like(qs[0]), Ks[0], Vs[0], 0, 1 / math.sqrt(hd))
        assert (got.double().cpu().view(-1, nh, hd) - expected).abs().max() <= BOUND


@pytest.mark.parametrize("nh,q_lens,ctx,page,sink", [
    (16, [1], [0], 16, False), (16, [128, 1], [0, 128], 16, True), (5, [129, 40], [127, 300], 8, False),
    (16, [513], [70], 16, True), (16, [64] * 9 + [300], [0, 20] * 5, 32, False), (2, [200], [1], 128, True)])
def test_rows_that_are_keys_and_values(ops, cuda_device, nh, q_lens, ctx, page, sink):
    from zephyr_b200.kernels.ops import kv_row_permutation

    hd, rank = 160, 128
    totals = [c + n for c, n in zip(ctx, q_lens)]
    pages = sum(-(-n // page) for n in totals) + 2
    table, tables = make_tables(totals, page, pages, 420)
    cache = torch.full((pages, page, hd), float("nan"), dtype=torch.bfloat16)
    rows, qs = [], []
    for r, total in enumerate(totals):
        rows.append(rand((total, hd), torch.bfloat16, "cpu", 421 + 3 * r))
        qs.append(rand((q_lens[r], nh, hd), torch.bfloat16, "cpu", 422 + 3 * r))
        for p in range(total):
            cache[tables[r][p // page], p % page] = rows[r][p][torch.argsort(kv_row_permutation(p, hd, torch.bfloat16))]
    cache = cache.view(pages, page * hd).to(cuda_device)
    q = torch.cat(qs).reshape(-1, nh * hd).to(cuda_device)
    sinks = rand((nh,), torch.float32, cuda_device, 7) if sink else None
    starts = torch.tensor([sum(q_lens[:r]) for r in range(len(q_lens))], dtype=torch.int32, device=cuda_device)
    lens, behind = (torch.tensor(v, dtype=torch.int32, device=cuda_device) for v in (q_lens, ctx))
    tiles = in_order_of_keys(tiles_for(q_lens, ops.paged_prefill_tile_tokens(), cuda_device), q_lens, ctx)
    status, before = ops.new_status(cuda_device), ops.LAUNCH_COUNTS.get("paged_prefill_tc", 0)
    got = ops.paged_prefill(q, cache, table.to(cuda_device), *tiles, starts, lens, behind, nh, 1, hd, 0, 1 / math.sqrt(hd), status,
                            torch.full_like(q, float("nan")), sinks=sinks, keys_only=True, value_dim=rank)
    ops.check_status(status)
    assert ops.LAUNCH_COUNTS["paged_prefill_tc"] == before + 1
    at = 0
    for r, n in enumerate(q_lens):
        kept = rows[r].unsqueeze(1)
        expected = plain(qs[r], kept, kept[..., :rank], ctx[r], 1 / math.sqrt(hd), sinks.cpu() if sink else None)
        assert (got[at:at + n].double().cpu().view(n, nh, hd)[..., :rank] - expected).abs().max() <= BOUND
        at += n


def test_a_prompt_beside_decoding_rows(ops, cuda_device, tmp_path):
    """Which form of a CTA a prompt's heads run in, and with that the last bits of the prompt's result, does not hang on the rows
    that only decode beside it."""
    from tiny_configs import tiny_config
    from zephyr_b200 import write_random_model
    from zephyr_b200.config import LayerCall, load_model_spec
    from zephyr_b200.engine import ModelRunner, StepEntry
    from zephyr_b200.parts import Model
    from zephyr_b200.weights import Checkpoint

    config = dataclasses.replace(tiny_config("A"), num_attention_heads=16, num_key_value_heads=8, head_dim=128, max_position_embeddings=4096)
    folder = write_random_model(config, 5, tmp_path / "model", dtype=torch.bfloat16)
    model = Model.load(load_model_spec(folder), Checkpoint(folder), torch.bfloat16, cuda_device)
    runner, mixer, tokens = ModelRunner(model, 16, 300, 16), model.layers[0].mixer, 2048
    projected = rand((tokens + 8, (16 + 2 * 8) * 128), torch.bfloat16, cuda_device, 530)
    results = []
    for beside in (0, 8):
        names = [f"{beside} {i}" for i in range(beside + 1)]
        for name in names:
            assert runner.add_request(name)
        ctx = runner.build_context([StepEntry(names[0], [1] * tokens)] + [StepEntry(name, [1]) for name in names[1:]])
        before = ops.LAUNCH_COUNTS.get("paged_prefill_tc", 0)
        results.append(mixer.core(projected[:tokens + beside], ctx, LayerCall(0, 0))[:tokens].clone())
        assert ops.LAUNCH_COUNTS["paged_prefill_tc"] == before + 1
    runner.check()
    assert torch.equal(*results)
