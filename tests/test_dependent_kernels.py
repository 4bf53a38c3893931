"""What kernels that start before the one in front of them has ended, and kernels whose copies run beside them, have to keep to, read
from the sources."""

import re

from zephyr_b200.kernels.build import SOURCE_DIR

# Written before any step, or by the kernel alone: the only pointers that may be declared free of other writers.
CONSTANT = {"table", "w", "bias", "q_norm_w", "k_norm_w", "cos_table", "sin_table"}
OWN = {"out", "q_out"}
# What kernels index ahead of their wait: arrays of their own (barriers, shared memory, registers), ...
LOCAL = {"consumed", "empty", "full", "own_full", "page_ids", "prefix", "qempty", "qfull", "trace", "plans", "place_empty", "place_full", "place_s",
         "half_of_row", "bars", "kv_empty", "kv_full", "note", "o_done", "p_full", "s_full", "red", "w_ok", "w_row", "x_ok", "x_row", "falling", "power",
         "wild", "wild_token", "smem", "smem_raw", "smem_unaligned", "f_smem_raw", "gs_smem", "gx_smem_raw", "gf_smem_raw"}
# ... the step's description, which lies there before its first kernel, weights, and the launch's own arguments.
GIVEN = {"paged_decode_kernel": {"a.block_table", "a.row_ctx", "a.row_q_start", "a.rows", "table", "x", "y"}, "fused_chain_kernel": {"a.map", "a.stage", "a.tiled"},
         "retention_tc_kernel": {"a.decay"}, "qk_norm_rope_cache_wide_kernel": {"positions", "token_row", "scale_x", "scale_y"}}


def kernels():
    """(file, name, parameters, body) of every kernel."""
    for path in sorted(SOURCE_DIR.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for found in re.finditer(r"__global__\s+void\s+(?:__cluster_dims__\([^)]*\)\s*)?(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
            depth, end = 1, found.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[end], 0)
                end += 1
            parameters, start = text[found.end():end - 1], text.index("{", end)
            depth, stop = 1, start + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[stop], 0)
                stop += 1
            yield path.name, found.group(1), [p.strip() for p in parameters.split(",")], text[start:stop]


def test_dependent_kernels_wait():
    """Every kernel that is launched as a dependent waits for the kernels before it."""
    text = "".join(path.read_text() for path in SOURCE_DIR.glob("*.cu"))
    launched = set(re.findall(r"launch_dependent\(\s*(\w+_kernel)\b", text)) | {"gemm_small_kernel", "gemm_tc_experts_kernel"}
    waiting = {name for _, name, _, body in kernels() if "wait_for_prior_grids()" in body}
    assert len(launched) > 20 and launched <= waiting


def test_dependent_kernels_do_not_declare_other_kernels_results_constant():
    dependent = [k for k in kernels() if "wait_for_prior_grids()" in k[3]]
    assert len(dependent) > 25
    for file, name, parameters, body in dependent:
        for parameter in parameters:
            if "__restrict__" in parameter:
                assert parameter.split()[-1].lstrip("*") in CONSTANT | OWN, (file, name, parameter)
        assert "__ldg(" not in body and ".nc." not in body, (file, name)


def test_dependent_kernels_index_nothing_of_other_kernels_ahead_of_their_wait():
    for file, name, _, body in kernels():
        if "wait_for_prior_grids()" not in body:
            continue
        several = name in ("paged_decode_kernel", "fused_chain_kernel")          # roles, each with a wait of its own
        ahead = body[:(body.index if several else body.rindex)("wait_for_prior_grids()")]
        indexed = set(re.findall(r"(?<![\w.])(?:a\.)?[A-Za-z_]\w*(?=\[)", ahead))
        assert indexed <= LOCAL | GIVEN.get(name, set()), (file, name, indexed - LOCAL)


def test_kernels_whose_wait_runs_out_let_their_copies_land():
    """A CTA that gives up leaves its shared memory to another one only behind its own copies."""
    copying = [k for k in kernels() if re.search(r"(bulk_copy_g2s|tiled_copy_2d_g2s(_pair)?)\(", k[3])]
    assert len(copying) >= 7
    for file, name, _, body in copying:
        assert "let_copies_land()" in body, (file, name)


def test_the_compiler_keeps_stores_in_front_of_fences_and_arrivals():
    """A fence, a wait or an arrival that does not name memory to the compiler lets it move plain stores and loads across."""
    ordering = re.compile(r"fence\.|mbarrier\.(?!init|test|try)|wait_group|barrier\.(cta|cluster)|\bbar\.sync|tcgen05\.(commit|wait|fence)|griddepcontrol\.")
    seen = 0
    for path in sorted(SOURCE_DIR.glob("*.cu*")):
        for statement in re.findall(r"asm volatile\((.*?)\);", re.sub(r"//[^\n]*", "", path.read_text()), re.S):
            if ordering.search(statement) and "complete_tx" not in statement:
                seen += 1
                assert '"memory"' in statement, (path.name, statement)
    assert seen > 20


def test_stores_for_a_pairs_tensor_cores_are_announced_within_their_own_cta():
    """Behind plain stores that the tensor cores are to read comes an arrival on a barrier of the same CTA: one on the other CTA's barrier is not
    ordered behind them."""
    seen = 0
    for file, name, _, body in kernels():
        for found in re.finditer(r"fence_proxy_async\(\);", body):
            arrival = re.search(r"\b(tc_mbar_arrive|mbar_arrive\w*|__syncthreads\w*|signal|bar_sync\w*)\(", body[found.end():])
            seen += 1
            assert arrival is None or arrival.group(1) not in ("mbar_arrive_at", "mbar_arrive_in_cluster"), (file, name)
    assert seen >= 5
