"""Rules of programmatic launches that no run can show to hold, read from the kernels' source."""
import os
import re

import pytest

from dualquant_b200 import build

CALL = "grid_dep_wait();"


def _kernels():
    """name -> (parameter list, body without comments) of every __global__ function"""
    found = {}
    for name in sorted(os.listdir(build.CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(build.CSRC, name)).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__\w+__\s*\((?:[^()]|\([^()]*\))*\)\s*)*(\w+)\s*\(([^{;]*?)\)\s*\{", text):
            depth, at = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            found[m.group(1)] = (m.group(2), text[m.end():at - 1])
    return found


KERNELS = _kernels()
STARTS_EARLY = sorted(k for k, (_, body) in KERNELS.items() if "grid_dep_launch_dependents" in body or CALL in body)
# Kernels whose first loads of what an earlier kernel wrote stand right behind the wait.  (The others' stand behind a barrier
# as well, whose phase the thread that has waited completes.)
READS_AT_ONCE = ("act_quant", "quant_fp4", "scale_cols", "codes_to", "expand_w", "rope_kv")
LOADS_ORDERED = READS_AT_ONCE + ("gemv_fused", "gemm_w4a4_e4m3", "gemm_a16w4", "gemm_fp4_persist", "column_stat",
                                 "iteration", "finish")


def test_the_kernels_are_found():
    assert len(KERNELS) >= 30 and len(STARTS_EARLY) >= 15
    assert {"act_quant_rows_kernel", "act_quant_had28_kernel", "expand_w_e4m3_kernel", "gemv_fused_kernel"} <= set(STARTS_EARLY)


@pytest.mark.parametrize("kernel", STARTS_EARLY)
def test_a_kernel_that_starts_the_next_one_early_waits_itself(kernel):
    """Only its own griddepcontrol.wait shows a kernel what the kernels before it wrote: each waits, in its own body, and
    the quantisers before all they read (that the kernel between has waited is no substitute)."""
    body = KERNELS[kernel][1]
    assert CALL in body
    if kernel.startswith(READS_AT_ONCE):
        before = body[: body.index(CALL)]
        assert before.count("{") == before.count("}"), "the wait is conditional"
        assert not re.search(r"\bif\s*\([^)]*\)\s*$", before), "the wait is conditional"


@pytest.mark.parametrize("kernel", [k for k in STARTS_EARLY if k.startswith(LOADS_ORDERED)])
def test_loads_behind_the_wait_are_ordinary_ones(kernel):
    """A `const __restrict__` parameter and __ldg say that the memory is constant while the kernel runs; the compiler may then
    place the load in front of the wait.  Only what the packed weight holds is read that way."""
    params, body = KERNELS[kernel]
    assert set(re.findall(r"const\s+[\w ]+\*\s*__restrict__\s+(\w+)", params)) <= {"w_packed", "sw_t"}
    assert set(re.findall(r"__ldg\((\w+)", body)) <= {"sw_row", "sxp"}  # sxp: behind the last group's barrier
