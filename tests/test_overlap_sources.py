"""Rules that every kernel whose start may overlap the end of the one in front of it keeps (csrc/lowbit_internal.h, launch_overlaps), read off
the sources: what breaks one of them shows on a GPU only when two blocks happen to meet on an SM, as a hang or as a stale value."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ipex_llm_b200", "csrc")


def closed(text, at, pair):
    """the place behind what closes the bracket in front of ``at``"""
    depth = 1
    while depth:
        depth += (text[at] == pair[0]) - (text[at] == pair[1])
        at += 1
    return at


def kernels():
    """parameters and body of every __global__ function that waits for, or releases, another launch"""
    for folder, _, names in os.walk(CSRC):
        for name in sorted(names):
            if not name.endswith((".cu", ".cuh")):
                continue
            text = re.sub(r"//[^\n]*", "", open(os.path.join(folder, name)).read())
            while (bounds := text.find("__launch_bounds__")) >= 0:
                text = text[:bounds] + text[closed(text, text.index("(", bounds) + 1, "()"):]
            for at in (m.start() for m in re.finditer(r"\b__global__\b", text)):
                head = re.compile(r"(\w+)\s*\(([^{;]*)\)\s*\{").search(text, at)
                if head is None:
                    continue
                end = closed(text, head.end(), "{}")
                if re.search("griddepcontrol|pdl_wait|pdl_release", text[head.end():end]):
                    yield pytest.param(head.group(2), text[head.end():end], id=f"{name}:{head.group(1)}")


KERNELS = list(kernels())


def test_the_kernels_are_found():
    assert {"exact_kernel", "split3_kernel", "pair_kernel", "skinny_kernel", "gemv_kernel", "sdp_fp8_prompt_kernel", "reduce_partials_kernel",
            "delta_walk_kernel"} <= {k.id.split(":")[1] for k in KERNELS}


@pytest.mark.parametrize("params,body", KERNELS)
def test_tensor_memory_is_held_before_dependents_may_start(params, body):
    """A dependent may allocate tensor memory in front of its wait.  Were it let onto an SM before this kernel's block there has its own, the
    one would wait for the other's columns and the other for the first one's end."""
    if "tcgen05.alloc" in body and "griddepcontrol.launch_dependents" in body:
        assert body.index("tcgen05.alloc") < body.index("griddepcontrol.launch_dependents")


@pytest.mark.parametrize("params,body", KERNELS)
def test_no_input_is_promised_to_be_constant(params, body):
    """What the launch in front leaves is written while the kernel already runs.  const __restrict__ says that it is not, and lets the
    compiler read it by the path for constants."""
    assert "__restrict__" not in params
