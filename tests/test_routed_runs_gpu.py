"""The routed feed-forward's tcgen05 products over runs of an expert's tokens, at the edges of runs, of blocks of 128 matrix rows
and of steps along K, against plain float64 experts."""

import pytest
import torch

from test_kernels_gpu import ops  # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu
F64 = torch.float64


def plain(x, ids, weights, gate, up, down, act, weigh_inputs):
    out = torch.zeros(x.shape[0], down.shape[1], dtype=F64)
    for e in range(gate.shape[0]):
        for j in range(ids.shape[1]):
            t = (ids[:, j] == e).nonzero().flatten()
            h, w = x[t].double(), weights[t, j].double().unsqueeze(1)
            g, u = h @ gate[e].double().T, h @ up[e].double().T
            if weigh_inputs:
                g, u = g * w, u * w
            hidden = ((g * torch.sigmoid(g) if act == "silu" else g.clamp(min=0)) * u).to(torch.bfloat16).double()
            y = (hidden @ down[e].double().T).to(torch.bfloat16).double()
            out.index_add_(0, t, y if weigh_inputs else y * w)
    return out


@pytest.mark.parametrize("counts,width,ff,act,weigh_inputs", [
    ([1], 64, 8, "silu", False), ([16, 0, 17, 1], 72, 24, "silu", False),        # widths that end inside a step along K
    ([64, 65, 63, 0, 2], 128, 72, "relu", False),                                # runs of up to 64, one of them cut in two
    ([100, 129, 40], 200, 136, "silu", True),                                    # 272 rows of gates and ups: a block of 16 rows
    ([128, 0, 0, 257], 136, 64, "silu", False),
    ([700, 0, 3, 256, 257, 15], 256, 128, "relu", True), ([0, 513], 1024, 200, "silu", False)])
def test_runs_of_tokens(ops, cuda_device, counts, width, ff, act, weigh_inputs):
    g = torch.Generator().manual_seed(31)
    E, T = len(counts), sum(counts)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(T, generator=g)].to(torch.int32).view(T, 1)
    x = torch.randn(T, width, generator=g).bfloat16()
    gate, up = (((torch.randn(E, ff, width, generator=g)) * width ** -0.5).bfloat16() for _ in range(2))
    down = (torch.randn(E, width, ff, generator=g) * ff ** -0.5).bfloat16()
    weights = torch.rand(T, 1, generator=g) + 0.5
    both = ops.interleave_gate_up(gate.to(cuda_device), up.to(cuda_device))
    before = ops.LAUNCH_COUNTS.get("gemm_tc_grouped", 0)
    got = ops.routed_experts(x.to(cuda_device), ids.to(cuda_device), weights.to(cuda_device), both, None, down.to(cuda_device), act=act,
                             weigh_inputs=weigh_inputs).cpu().double()
    ops.check_status(ops.device_status(cuda_device))
    assert ops.LAUNCH_COUNTS["gemm_tc_grouped"] == before + 2
    expected = plain(x, ids, weights, gate, up, down, act, weigh_inputs)
    # The hidden values, the expert's output and the sum are rounded to bfloat16, 2^-9 each.
    assert (got - expected).abs().max() <= 2.0 ** -6 * max(1.0, float(expected.abs().max()))


def test_every_token_to_every_expert_and_to_none(ops, cuda_device):
    """Choices that name no expert's matrix, and more choices than runs hold."""
    g = torch.Generator().manual_seed(32)
    E, T, width, ff = 3, 90, 64, 32
    ids = torch.stack([torch.randperm(E + 2, generator=g) for _ in range(T)]).to(torch.int32)
    x = torch.randn(T, width, generator=g).bfloat16()
    gate, up, down = ((torch.randn(E, *s, generator=g) * 0.15).bfloat16() for s in ((ff, width), (ff, width), (width, ff)))
    weights = torch.rand(T, E + 2, generator=g)
    both = ops.interleave_gate_up(gate.to(cuda_device), up.to(cuda_device))
    got = ops.routed_experts(x.to(cuda_device), ids.to(cuda_device), weights.to(cuda_device), both, None, down.to(cuda_device)).cpu().double()
    expected = plain(x, ids, weights, gate, up, down, "silu", False)
    for j in range(E + 2):
        t = (ids[:, j] >= E).nonzero().flatten()
        expected.index_add_(0, t, x[t].double() * weights[t, j].double().unsqueeze(1))       # an identity expert
    assert (got - expected).abs().max() <= 2.0 ** -6 * max(1.0, float(expected.abs().max()))


@pytest.mark.parametrize("rows,outputs,k", [(65, 18, 2048), (66, 1, 64), (777, 24, 1000), (2049, 9, 72), (5000, 3, 264), (4097, 16, 64)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_many_rows_and_few_outputs(ops, cuda_device, rows, outputs, k, out_dtype):
    g = torch.Generator().manual_seed(33)
    wide = torch.randn(rows, k + 8, generator=g).bfloat16().to(cuda_device)
    x, w = wide[:, :k], (torch.randn(outputs, k, generator=g) * k ** -0.5).bfloat16().to(cuda_device)     # rows further apart than they are long
    before = ops.LAUNCH_COUNTS.get("gemm_small", 0)
    got = ops.linear(x, w, out_dtype=out_dtype)
    assert ops.LAUNCH_COUNTS.get("gemm_small", 0) - before == int(rows <= 4096 or outputs % 8 != 0)
    expected = x.double() @ w.double().T
    # float32: k sums of products of about k^-1/2; bfloat16 rounds values of up to six.
    assert got.dtype == out_dtype and (got.double() - expected).abs().max() <= (2.0 ** -6 if out_dtype == torch.bfloat16 else 2e-5)


@pytest.mark.parametrize("outputs,k", [(18, 2048), (18, 4096), (9, 1000), (24, 256), (1, 7168)])
def test_a_routers_logits_do_not_depend_on_the_step(ops, cuda_device, outputs, k):
    """The same bits for a row in a step of a few tokens and of many."""
    g = torch.Generator().manual_seed(34)
    x, w = torch.randn(6000, k, generator=g).bfloat16().to(cuda_device), (torch.randn(outputs, k, generator=g) * k ** -0.5).bfloat16().to(cuda_device)
    few = ops.linear(x[:8], w, out_dtype=torch.float32)
    for rows in (65, 333, 777, 1000) if outputs % 8 == 0 else (65, 777, 2049, 4100, 6000):
        before = ops.LAUNCH_COUNTS.get("gemm_small", 0)
        got = ops.linear(x[:rows], w, out_dtype=torch.float32)
        assert ops.LAUNCH_COUNTS["gemm_small"] == before + 1 and torch.equal(got[:8], few), rows


@pytest.mark.parametrize("outputs,rows,own", [(16, 1024, True), (16, 1025, False), (24, 2048, False), (8, 2048, True), (8, 2049, False),
                                              (18, 6144, True), (18, 6145, False), (25, 65, False)])
def test_where_a_routers_product_runs(ops, cuda_device, outputs, rows, own):
    """On the few-row kernel while the library's product is the slower one."""
    g = torch.Generator().manual_seed(35)
    x, w = torch.randn(rows, 256, generator=g).bfloat16().to(cuda_device), torch.randn(outputs, 256, generator=g).bfloat16().to(cuda_device)
    before = ops.LAUNCH_COUNTS.get("gemm_small", 0)
    got = ops.linear(x, w, out_dtype=torch.float32)
    assert ops.LAUNCH_COUNTS.get("gemm_small", 0) - before == int(own)
    # float32 sums of 256 products of about one.
    assert (got.double() - x.double() @ w.double().T).abs().max() <= 256 * 2.0 ** -20


def test_rows_that_share_memory(ops, cuda_device):
    """One row seen as many, and rows that overlap, whatever kernel the number of outputs asks for."""
    g = torch.Generator().manual_seed(36)
    one, run, w = (torch.randn(*shape, generator=g).bfloat16().to(cuda_device) for shape in ((1, 64), (64 + 8 * 99,), (9, 64)))
    for x in (one.expand(100, 64), run.as_strided((100, 64), (8, 1))):
        for weight in (w, w[:1].expand(9, 64)):
            got = ops.linear(x, weight, out_dtype=torch.float32)
            # float32 sums of 64 products of about one.
            assert (got.double() - x.double() @ weight.double().T).abs().max() <= 64 * 2.0 ** -20
