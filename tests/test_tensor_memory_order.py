"""Tensor-memory stores are waited for before their columns are freed.

tcgen05.st is asynchronous and tcgen05.dealloc does not wait for it: a block
resident beside the freeing one may be given the columns at once, so a store
still under way would land in that block's z-flux ring.  The order is read
from the source: every wait the last store needs has to stand between it and
the barrier in front of the deallocation."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "muram_main_gb300", "csrc")


def _kernel_body(path, name):
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, path)).read())
    at = src.index("{", re.search(r"\b%s\(" % name, src).end())
    depth = 0
    for i in range(at, len(src)):
        depth += (src[i] == "{") - (src[i] == "}")
        if depth == 0:
            return src[at : i + 1]
    raise AssertionError(f"{name}: unbalanced braces")


def test_stage_kernel_waits_for_its_stores_before_freeing():
    body = _kernel_body("gpumhd_stage_tm.cuh", "k_stage_tm")
    last_store = body.rindex("tm_store12(")
    free = body.index("tm::tmem_dealloc(")
    barrier = body.rindex("tm::tc_fence_before()", 0, free)
    assert last_store < barrier
    assert "tm::tmem_wait_st()" in body[last_store:barrier]
