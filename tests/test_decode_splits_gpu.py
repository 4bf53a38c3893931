"""How a decode step cuts its contexts: the same attention whether a context is one item or many, at the edges of tiles and of the
rule's lines."""

import math

import pytest
import torch

from test_kernels_gpu import build_paged_case, ops, rand  # noqa: F401  (ops: a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,nkv,context,whole", [(1, 8, 256, True), (1, 8, 288, False), (8, 8, 2208, True), (8, 8, 2240, False),
                                                    (12, 8, 4096, True), (12, 8, 4097, False), (37, 4, 100, True), (40, 4, 100, False)])
def test_the_rule(ops, cuda_device, rows, nkv, context, whole):
    if ops._sm_count() != 148:
        pytest.skip("lines of a GPU with 148 SMs")
    split = ops.decode_split_size(rows, nkv, context)
    assert (split >= context) == whole
    assert split % 32 == 0


@pytest.mark.parametrize("nh,nkv,ctx,window,sink", [
    (16, 8, [0, 31, 32, 33, 300, 1, 63, 64], 0, False), (16, 8, [169] * 9 + [5, 511], 0, True),
    (8, 2, [1000, 3, 77, 500, 31, 32, 900, 12, 13, 14, 15, 16, 17, 18, 19, 20, 21, 22, 23, 24], 0, False),
    (16, 8, [700, 699, 20, 64, 65, 66, 67], 100, False)])
def test_whole_contexts(ops, cuda_device, nh, nkv, ctx, window, sink):
    hd, n = 128, len(ctx)
    q, cache, meta, Ks, Vs, qs = build_paged_case(cuda_device, torch.bfloat16, nh, nkv, hd, 16, [1] * n, ctx, 500)
    rows, sinks = torch.arange(n, dtype=torch.int32, device=cuda_device), torch.linspace(-1, 2, nh, device=cuda_device) if sink else None
    status = ops.new_status(cuda_device)
    assert ops.decode_split_size(n, nkv, max(ctx) + 1, min(max(ctx) + 1, window or 1 << 30)) >= max(ctx) + 1        # one item each
    got = {}
    for split in (None, 0, 128):
        got[split] = ops.paged_decode(q, cache, meta["table"], rows, meta["row_q_start"], meta["row_ctx"], max(ctx) + 1, nh, nkv, hd, window,
                                      1 / math.sqrt(hd), status, torch.full_like(q, float("nan")), split_size=split, sinks=sinks)
    ops.check_status(status)
    for r in range(n):
        lo = max(0, ctx[r] + 1 - window) if window else 0
        for h in range(nh):
            s = qs[r][0, h].double() @ Ks[r][lo:, h // (nh // nkv)].double().T / math.sqrt(hd)
            if sink:
                s = torch.cat([s, sinks[h].cpu().double().view(1)])
            expected = torch.softmax(s, -1)[:ctx[r] + 1 - lo] @ Vs[r][lo:, h // (nh // nkv)].double()
            # Weights and the result are rounded to bfloat16, 2^-9 each of values up to four.
            for split in got:
                assert (got[split][r].double().cpu().view(nh, hd)[h] - expected).abs().max() <= 3.2e-2, (split, r, h)


@pytest.mark.parametrize("ctx,bound,window,whole", [
    ([169] * 12, 4096, 0, True), ([1000] * 6 + [1020] * 6, 1024, 0, True), ([700, 690, 20, 640, 64, 650], 1024, 0, True),
    ([4095] + [99] * 11, 4096, 0, False), ([20] * 12 + [3999], 4096, 0, False), ([1999] + [99] * 7, 2000, 0, False),
    ([4095] + [99] * 11, 4096, 100, True)])
def test_contexts_of_unequal_lengths(ops, cuda_device, ctx, bound, window, whole):
    """One item a (row, key/value head) pair while the contexts are near each other in length; spread over all CTAs where one CTA would
    stream on alone.  The lengths, not the bound on them that a captured step knows, decide."""
    nh, nkv, hd, n = 16, 8, 128, len(ctx)
    q, cache, meta, Ks, Vs, qs = build_paged_case(cuda_device, torch.bfloat16, nh, nkv, hd, 16, [1] * n, ctx, 520)
    rows, status, out = torch.arange(n, dtype=torch.int32, device=cuda_device), ops.new_status(cuda_device), torch.full_like(q, float("nan"))
    trace = torch.zeros((1024, 8), dtype=torch.int32, device=cuda_device)
    ops.paged_decode_trace(trace)
    for _ in range(2):                   # (the counters are left as they were found)
        ops.paged_decode(q, cache, meta["table"], rows, meta["row_q_start"], meta["row_ctx"], bound, nh, nkv, hd, window, 1 / math.sqrt(hd),
                         status, out)
    ops.paged_decode_trace(None)
    ops.check_status(status)
    lo = [max(0, c + 1 - window) if window else 0 for c in ctx]
    tiles = [-(-(c + 1) // 32) - l // 32 for c, l in zip(ctx, lo)]
    most = max(tiles) if whole else -(-sum(tiles) * nkv // ops._sm_count())
    assert int(trace[:, 6].max()) == most                             # tiles of the CTA that has the most
    for r in range(n):
        for h in range(nh):
            s = qs[r][0, h].double() @ Ks[r][lo[r]:, h // 2].double().T / math.sqrt(hd)
            expected = torch.softmax(s, -1) @ Vs[r][lo[r]:, h // 2].double()
            # Weights and the result are rounded to bfloat16, 2^-9 each of values up to four.
            assert (out[r].double().cpu().view(nh, hd)[h] - expected).abs().max() <= 3.2e-2, (r, h)


@pytest.mark.parametrize("options,size,most", [
    (["--batch", "12", "--context", "170", "--split", "0"], "balanced", 4),         # 12 rows x 8 heads x 6 tiles over 148 CTAs
    (["--batch", "12", "--context", "170"], "chosen", 6), (["--batch", "12", "--context", "170", "--split", "64"], 64, 4),     # (two items of two tiles)
    (["--contexts", "4096,100,100,100,100,100"], "chosen", 8), (["--contexts", "4096,100,100,100,100,100", "--split", "4096"], 4096, 128)])
def test_the_timing_program_cuts_as_it_says(ops, cuda_device, capsys, options, size, most):
    import json

    from zephyr_b200.kernels import timing

    timing.main(["decode_attention", "--warmup", "1", "--iters", "2", *options])
    line = json.loads(capsys.readouterr().out)
    assert line["split_size"] == size and line["timeline_ns"]["tiles"][1] == most


@pytest.mark.parametrize("even", [True, False])
@pytest.mark.parametrize("form", ["narrow heads", "keys that are values", "distance bias", "bounded scores", "a chunk", "norms inside"])
def test_the_cut_by_lengths_in_every_form(ops, cuda_device, form, even):
    """The kernel that looks at the lengths gives what the cut that it takes gives on its own, bit for bit."""
    hd, page, n = 64 if form == "narrow heads" else 128, 16, 12
    nh, nkv = (48, 8) if form == "distance bias" else (16, 8)
    ctx = [400 + 7 * r for r in range(n)] if even else [3800] + [40 + 9 * r for r in range(n - 1)]
    keys_only, chunk = form == "keys that are values", 4000 if form == "a chunk" else 0
    pages = [-(-(c + 1) // page) for c in ctx]
    table, at = torch.zeros((n, max(pages)), dtype=torch.int32), 1
    order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(3)) + 1
    for r, count in enumerate(pages):
        table[r, :count], at = order[at - 1:at - 1 + count], at + count
    table = table.to(cuda_device)
    shape = (sum(pages) + 1, nkv * page * hd) if keys_only else (sum(pages) + 1, 2, nkv, page, hd)
    cache = rand(shape, torch.bfloat16, cuda_device, 540)
    rows, behind = torch.arange(n, dtype=torch.int32, device=cuda_device), torch.tensor(ctx, dtype=torch.int32, device=cuda_device)
    status, most = ops.new_status(cuda_device), max(ctx) + 1
    options = {"distance bias": dict(distance_bias=(torch.linspace(0.1, 2, nh, device=cuda_device), torch.linspace(0.01, 0.5, nh, device=cuda_device))),
               "bounded scores": dict(softcap=20.0, sinks=torch.linspace(-1, 2, nh, device=cuda_device))}.get(form, {})
    if chunk:
        options["chunk"] = chunk
    got = {}
    for split in (None, 4096 if even else 0):
        out = torch.full((n, nh * hd), float("nan"), dtype=torch.bfloat16, device=cuda_device)
        if form == "norms inside":
            scale = rand((hd,), torch.float32, cuda_device, 541).to(torch.bfloat16)
            qkv = rand((n, (nh + 2 * nkv) * hd), torch.bfloat16, cuda_device, 542)
            ops.paged_decode_fused(qkv, cache, table, rows, rows, behind, most, nh, nkv, hd, 0, hd ** -0.5, scale, scale, 1e-6, None, None,
                                   status, out, split_size=split)
        else:
            q = rand((n, nh * hd), torch.bfloat16, cuda_device, 543)
            ops.paged_decode(q, cache, table, rows, rows, behind, most, nh, nkv, hd, 0, hd ** -0.5, status, out, split_size=split,
                             keys_only=keys_only, **options)
        got[split] = out
    ops.check_status(status)
    chosen, alone = got.values()
    assert torch.isfinite(chosen).all() and torch.equal(chosen, alone)
