"""What a kernel may do before the one behind it is allowed to start, read from the sources: no GPU runs code that waits for good."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jacobiforcing_b200", "csrc")
ALLOC = re.compile(r"tcgen05\.alloc|\btmem_alloc\(")
TRIGGER = re.compile(r"\bpdl_trigger\(\)|\bpdl_begin\(\)|griddepcontrol\.launch_dependents")
BARRIER = re.compile(r"__syncthreads\(\)|tp_cluster_sync\(\)")


def kernels():
    """(file, name, body) of every __global__ function, comments taken out."""
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        src = re.sub(r"__(?:launch_bounds|cluster_dims)__\s*\([^()]*\)", "", src)
        for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\((?:[^;{}]|\{\})*?\)\s*\{", src):
            depth, at = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(src[at], 0)
                at += 1
            yield f, m.group(1), src[m.end():at]


ALLOCATING = [(f, n, b) for f, n, b in kernels() if ALLOC.search(b)]


def test_the_allocating_kernels_are_found():
    assert {n for _, n, _ in ALLOCATING} >= {"pair_kernel", "flash_kernel"}


@pytest.mark.parametrize("name,body", [(n, b) for _, n, b in ALLOCATING], ids=[n for _, n, _ in ALLOCATING])
def test_dependents_start_behind_the_allocation_of_tensor_memory(name, body):
    """A dependent that started earlier could take this block's columns and keep them until this grid ends, for which this block would
    have to get them: the trigger stands behind the allocation and a barrier that every warp passes after it."""
    triggers = [m.start() for m in TRIGGER.finditer(body)]
    if not triggers:
        return                                               # never lets a dependent start early
    last_alloc = max(m.end() for m in ALLOC.finditer(body))
    barrier = BARRIER.search(body, last_alloc)
    assert barrier and min(triggers) > barrier.end(), name
    if "cta_group::2" in body[:last_alloc]:                   # both CTAs of a pair
        pair = body.index("tp_cluster_sync()", last_alloc)
        assert min(triggers) > pair, name


def test_scores_wait_for_the_product_that_reads_the_weights_in_their_place():
    """Both lie in the same columns, and products with unlike accumulators are not promised to run in the order of their issue."""
    body = next(b for _, n, b in kernels() if n == "flash_kernel")
    output, scores = body.index("umma_bf16_ts("), body.index("umma_bf16(tm,")
    over = re.search(r"umma_commit\(&sm->(\w+)\[", body[output:scores])
    assert output < scores and over, "the product of the output is committed before the scores are issued"
    assert re.search(r"fl_wait\(&sm->%s\[" % over.group(1), body[output + over.end():scores])
