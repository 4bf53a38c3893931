"""The prompt kernel on tcgen05 with a window that keeps the first tokens and with a chunked mask, at the edges of its tiles of
128 keys, against a plain float64 attention and against the mma.sync kernel."""

import math

import pytest
import torch

from test_kernels_gpu import build_paged_case, ops, rand, tiles_for  # noqa: F401  (ops: a fixture)

pytestmark = pytest.mark.gpu


def plain(q, K, V, ctx, nh, nkv, window, keep, chunk, sinks, softcap):
    T = q.shape[0]
    i, j = torch.arange(ctx, ctx + T)[:, None], torch.arange(ctx + T)[None, :]
    seen = j <= i
    if window:
        seen = seen & (i - j < window)
    if chunk:
        seen = seen & (i // chunk == j // chunk)
    seen = seen | ((j <= i) & (j < keep))                  # kept first tokens stay through either mask
    out = []
    for h in range(nh):
        s = q[:, h].double() @ K[:, h // (nh // nkv)].double().T / math.sqrt(128)
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(~seen, -math.inf)
        if sinks is not None:
            s = torch.cat([s, sinks[h].double().expand(T, 1)], dim=1)
        out.append(torch.softmax(s, -1)[:, :ctx + T] @ V[:, h // (nh // nkv)].double())
    return torch.stack(out, 1)


@pytest.mark.parametrize("window,keep,chunk,softcap,sink,page", [
    (100, 1, 0, 0.0, False, 16), (64, 64, 0, 0.0, True, 16), (200, 128, 0, 0.0, False, 8), (130, 129, 0, 0.0, True, 32),
    (1, 300, 0, 0.0, False, 16), (300, 70, 0, 20.0, True, 16), (1000, 64, 0, 0.0, False, 16), (0, 0, 100, 0.0, True, 16),
    (0, 0, 128, 0.0, False, 16), (90, 0, 256, 0.0, False, 64), (60, 40, 200, 0.0, False, 16)])
def test_kept_windows_and_chunks(ops, cuda_device, window, keep, chunk, softcap, sink, page):
    nh, nkv, hd, q_lens, ctx = 4, 2, 128, [37, 300, 2, 129, 128], [0, 5, 400, 255, 256]
    q, cache, meta, Ks, Vs, qs = build_paged_case(cuda_device, torch.bfloat16, nh, nkv, hd, page, q_lens, ctx, 300)
    sinks = rand((nh,), torch.float32, cuda_device, 5) if sink else None
    status, got = ops.new_status(cuda_device), {}
    for tcgen05 in (True, False):
        ops.USE_TCGEN05_PREFILL = tcgen05
        before = ops.LAUNCH_COUNTS.get("paged_prefill_tc", 0)
        try:
            got[tcgen05] = ops.paged_prefill(q, cache, meta["table"], *tiles_for(q_lens, ops.paged_prefill_tile_tokens(), cuda_device),
                                             meta["row_q_start"], meta["row_q_len"], meta["row_ctx"], nh, nkv, hd, window,
                                             1 / math.sqrt(hd), status, torch.empty_like(q), chunk=chunk, sinks=sinks,
                                             softcap=softcap, keep_first=keep)
        finally:
            ops.USE_TCGEN05_PREFILL = True
        assert ops.LAUNCH_COUNTS.get("paged_prefill_tc", 0) - before == int(tcgen05)      # each ran on the kernel it is about
    ops.check_status(status)
    # Weights and the result are rounded to bfloat16 (2^-9 each, of values around one to four).
    assert (got[True].float() - got[False].float()).abs().max() <= 3 * 2.0 ** -7
    cursor = 0
    for r, n in enumerate(q_lens):
        expected = plain(qs[r], Ks[r], Vs[r], ctx[r], nh, nkv, window, keep, chunk, sinks.cpu() if sink else None, softcap)
        assert (got[True][cursor:cursor + n].double().cpu().view(n, nh, hd) - expected).abs().max() <= 1.6e-2 * 2
        cursor += n


@pytest.mark.parametrize("lengths,tcgen05", [([2], False), ([64], False), ([65], True), ([8] * 9, False), ([8] * 10, True), ([30, 200], True)])
@pytest.mark.parametrize("kind", ["kept", "latent"])
def test_short_prompts(ops, cuda_device, kind, lengths, tcgen05):
    """Prompts within one step of its keys that give every head an SM of its own run on the mma.sync kernel."""
    from zephyr_b200.config import FekotarConfig, TedulornConfig
    from zephyr_b200.engine import ModelRunner, StepEntry
    from zephyr_b200.parts import Model, expected_weights

    rot = {"base": 10000.0, "dims": 32}
    if kind == "kept":
        mixer = dict(heads=16, kv_heads=8, dim=128, vdim=128, scale=128 ** -0.5, v_mix=False, rot=rot, mask={"size": 40, "keep_first": 16})
        config = TedulornConfig(vocab=64, width=64, norm_eps=1e-6, embedding_scale=1.0, side_dim=0,
                                layers=({"type": "attention", "mixer": mixer, "mlp": None},))
    else:
        mixer = dict(heads=16, dim=64, rot_dim=32, vdim=64, kv_rank=128, q_rank=64, scale=160 ** -0.5, rot=rot)
        config = FekotarConfig(vocab=64, width=64, norm_eps=1e-6, logit_scale=1.0, bigram=None,
                               layers=({"type": "latent_attention", "mixer": mixer, "mlp": None},))
    spec = config.to_model_spec()
    expected = expected_weights(spec)

    class Store:
        def names(self):
            return tuple(expected)

        def shape(self, name):
            return tuple(expected[name].shape)

        def dtype(self, name):
            return torch.bfloat16

        def read(self, name):
            return rand(self.shape(name), torch.bfloat16, cuda_device, len(name)) * 0.1 + float(expected[name].role == "norm")

    model = Model.load(spec, Store(), torch.bfloat16, cuda_device)
    runner, call, got = ModelRunner(model, 16, 64, 16), spec.run_order[0], {}
    for row, n in enumerate(lengths):
        assert runner.add_request(row, n)
    x = rand((sum(lengths), 64), torch.bfloat16, cuda_device, 9)
    for own in (True, False):
        ctx = runner.build_context([StepEntry(row, [0] * n) for row, n in enumerate(lengths)])
        before = ops.LAUNCH_COUNTS.get("paged_prefill_tc", 0)
        ops.USE_TCGEN05_PREFILL = own
        try:
            got[own] = model.layers[0].mixer.forward(x, ctx, call).float()
        finally:
            ops.USE_TCGEN05_PREFILL = True
        assert ops.LAUNCH_COUNTS.get("paged_prefill_tc", 0) - before == int(own and tcgen05)
    runner.check()
    # The two kernels round probabilities and results to bfloat16, 2^-9 of them each, ahead of one more product.
    assert (got[True] - got[False]).abs().max() <= 2.0 ** -6 * float(got[False].abs().max())


@pytest.mark.parametrize("window,keep,chunk,bias,page", [
    (100, 40, 0, False, 16), (64, 64, 0, False, 8), (300, 130, 0, False, 16), (60, 40, 200, False, 16), (0, 0, 100, False, 16),
    (0, 0, 128, False, 32), (0, 0, 0, True, 16), (150, 0, 0, True, 64)])
@pytest.mark.parametrize("heads", ["in pairs", "singly"])
def test_masks_in_both_forms_of_a_cta(ops, cuda_device, heads, window, keep, chunk, bias, page):
    """Kept tokens, chunks and a distance bias with two heads a CTA and with one whose tiles of keys two slots share."""
    hd = 128
    nh, nkv = (32, 8) if heads == "in pairs" else (4, 2)
    q_lens, ctx = [130, 1, 127, 128, 90, 257], [0, 511, 129, 128, 64, 300]        # 9 tiles of 6 rows: 288 (head, tile) or 36
    q, cache, meta, Ks, Vs, qs = build_paged_case(cuda_device, torch.bfloat16, nh, nkv, hd, page, q_lens, ctx, 310)
    sinks = rand((nh,), torch.float32, cuda_device, 6)
    r1, r2 = (torch.linspace(0.1, 2.0, nh), torch.linspace(0.01, 0.5, nh)) if bias else (None, None)
    status, before = ops.new_status(cuda_device), ops.LAUNCH_COUNTS.get("paged_prefill_tc", 0)
    got = ops.paged_prefill(q, cache, meta["table"], *tiles_for(q_lens, ops.paged_prefill_tile_tokens(), cuda_device), meta["row_q_start"],
                            meta["row_q_len"], meta["row_ctx"], nh, nkv, hd, window, 1 / math.sqrt(hd), status, torch.full_like(q, float("nan")),
                            chunk=chunk, sinks=sinks, keep_first=keep,
                            distance_bias=(r1.to(cuda_device), r2.to(cuda_device)) if bias else None)
    ops.check_status(status)
    assert ops.LAUNCH_COUNTS["paged_prefill_tc"] == before + 1
    at = 0
    for r, n in enumerate(q_lens):
        if bias:
            i, j = torch.arange(ctx[r], ctx[r] + n)[:, None], torch.arange(ctx[r] + n)[None, :]
            seen, expected = (j <= i) & ((i - j < window) if window else (j <= i)), []
            for h in range(nh):
                s = qs[r][:, h].double() @ Ks[r][:, h // (nh // nkv)].double().T / math.sqrt(hd) - r1[h].double() * torch.log1p(
                    r2[h].double() * (i - j).clamp(min=0))
                s = torch.cat([s.masked_fill(~seen, -math.inf), sinks[h].cpu().double().expand(n, 1)], dim=1)
                expected.append(torch.softmax(s, -1)[:, :-1] @ Vs[r][:, h // (nh // nkv)].double())
            expected = torch.stack(expected, 1)
        else:
            expected = plain(qs[r], Ks[r], Vs[r], ctx[r], nh, nkv, window, keep, chunk, sinks.cpu(), 0.0)
        # Weights and the result are rounded to bfloat16 (2^-9 each, of values of up to four).
        assert (got[at:at + n].double().cpu().view(n, nh, hd) - expected).abs().max() <= 3.2e-2
        at += n
