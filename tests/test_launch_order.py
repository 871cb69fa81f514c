"""Programmatic dependent launches, read from the kernel sources.

A kernel that is launched as a programmatic dependent runs beside the kernel before it until
its own griddepcontrol.wait.  What it reads before that wait is stored by kernels that have
completed, but only the wait itself makes their stores visible to plain loads, which may be
answered from an L1 line of an earlier call.  A run cannot be relied on to show a stale read, so
the rule is checked where it is written."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpt-oss-amd_b200", "csrc")


def kernel_body(file, name):
    with open(os.path.join(CSRC, file)) as f:
        src = f.read()
    src = re.sub(r"//[^\n]*", "", src)
    start = re.search(r"__launch_bounds__\([^)]*\)\s*" + name + r"\(", src).start()
    start = src.index("{", start)
    depth, i = 0, start
    while True:
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        if depth == 0:
            return src[start:i + 1]
        i += 1


def loads(text, name):
    """Every use of the pointer `name` that reads through it: a subscript, or inside ld_l2()."""
    plain = re.findall(r"(?<!\w)" + name + r"\s*\[", text)
    l2 = re.findall(r"ld_l2\(\s*" + name + r"(?!\w)", text)
    return len(plain), len(l2)


@pytest.mark.parametrize("name", ["topk_i", "slot_of", "topk_w"])
def test_combine_reads_the_routing_past_l1(name):
    body = kernel_body("plan.cuh", "combine_kernel")
    before = body[:body.index("pdl_wait()")]
    assert loads(before, name) == (0, 1)


@pytest.mark.parametrize("name", ["g_off", "g_cnt", "g_tile_start"])
def test_down_gemm_reads_the_plan_past_l1(name):
    """The table copy sits behind `if (MODE == 0) pdl_wait()`: in the down launch no wait precedes it."""
    body = kernel_body("gemm_tc5_ts.cuh", "expert_gemm_ts_kernel")
    assert loads(body, name) == (0, 1)


@pytest.mark.parametrize("file,name", [
    ("plan.cuh", "permute_kernel"),
    ("route.cuh", "front_small_kernel"),
    ("gemm_tc5_ts.cuh", "expert_gemm_ts_kernel"),
    ("gemm_tc5_pair.cuh", "expert_gemm_pair_kernel"),
    ("plan.cuh", "combine_kernel"),
])
def test_trigger_follows_the_wait(file, name):
    """From the permute on: that a kernel has started then says that every kernel before its
    predecessor is complete, which the reads ahead of the wait rest on."""
    body = kernel_body(file, name)
    calls = re.findall(r"pdl_(wait|trigger)\(\)", body)
    assert "trigger" in calls
    for i, c in enumerate(calls):
        if c == "trigger":
            assert i > 0 and calls[i - 1] == "wait", calls
