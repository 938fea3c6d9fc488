"""Kernels that may be launched chained (they begin while their predecessor still writes what they read) must not promise the
compiler that anything they read is constant for their whole life: no ``__restrict__`` parameter, no ``__ldg``.  Read from the
source, since a load that the compiler moved over the wait shows in no result that a test could rely on."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "moe-explore_b200", "csrc")


def _kernels():
    """(name, parameters, body) of every __global__ function that waits for a predecessor."""
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"__global__ void\s+(?:__launch_bounds__\([^)]*\)\s+)?(\w+)\(", text):
            body = text.index("\n}", m.end())
            head, _, rest = text[m.end():body].partition(") {")
            if "grid_wait()" in rest:
                found.append((m.group(1), head, rest))
    return found


def test_the_chained_kernels_are_found():
    names = {name for name, _, _ in _kernels()}
    assert names == {"grouped_gemm_kernel", "copy_rows_kernel", "dispatch_rows_kernel", "combine_topk_kernel",
                     "combine_bwd_tokens_kernel", "router_backward_kernel"}


@pytest.mark.parametrize("name,params,body", _kernels(), ids=lambda v: v if v.isidentifier() else "")
def test_no_promise_of_constant_memory(name, params, body):
    assert "__restrict__" not in params
    assert "__ldg" not in body


def test_the_tile_walk_of_the_gemm_reads_its_maps_with_ordinary_loads():
    with open(os.path.join(CSRC, "gemm_kernel.cuh")) as f:
        assert "__ldg" not in f.read()
