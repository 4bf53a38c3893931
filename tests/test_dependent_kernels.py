"""What kernels that start before the one in front of them has ended, and kernels whose copies run beside them, have to keep to, read
from the sources."""

import re

from zephyr_b200.kernels.build import SOURCE_DIR

# Written before any step, or by the kernel alone: the only pointers that may be declared free of other writers.
CONSTANT = {"table", "w", "bias", "q_norm_w", "k_norm_w", "cos_table", "sin_table"}
OWN = {"out", "q_out"}


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


def test_kernels_whose_wait_runs_out_let_their_copies_land():
    """A CTA that gives up leaves its shared memory to another one only behind its own copies."""
    copying = [k for k in kernels() if re.search(r"(bulk_copy_g2s|tiled_copy_2d_g2s(_pair)?)\(", k[3])]
    assert len(copying) >= 7
    for file, name, _, body in copying:
        assert "let_copies_land()" in body, (file, name)
