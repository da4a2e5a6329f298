"""Kernels launched with programmatic serialization are resident while the kernel before them still writes: the pointers
through which they read that memory are handed to their wait, and are not declared __restrict__ (read from the source:
the qualifier's effect is the compiler's choice and cannot be provoked)."""
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = open(os.path.join(ROOT, "three-virtual-geometry_b200", "csrc", "vgcut_kernels.cu")).read()

# kernel -> what the kernel launched before it writes and it reads (vgc_cut's and vgc_cut_noalloc's sequences, HZB builds)
WRITTEN_BEFORE = {
    "k_reset": {"views"},  # k_noalloc_store_view
    "k_hzb_stream": {"plan"},  # k_reset
    "k_cells": {"views", "scenes"},  # k_reset
    "k_instances": {"units", "words"},  # k_cells (words: the control words it reads)
    "k_chunks": {"queue", "ctl"},  # k_instances
    "k_instances_redo": {"ctl"},  # k_chunks
    "k_budget": {"ctl"},  # k_instances_redo
    "k_finish": {"ctl"},  # k_instances_redo
    "k_retry": {"ctl"},  # k_finish
    "k_hzb_tiles": {"depth"},  # the caller's kernel that drew the image
    "k_hzb_tail": {"out"},  # k_hzb_tiles
}


def _kernel(name):
    m = re.search(r"__global__ void __launch_bounds__\([^{;]*?\)\s*%s\(" % name, SOURCE)
    assert m, name
    depth, end = 1, m.end()
    while depth:
        depth += {"(": 1, ")": -1}.get(SOURCE[end], 0)
        end += 1
    body = SOURCE[end:SOURCE.index("\n}\n", end)]
    return SOURCE[m.end():end - 1], body


@pytest.mark.parametrize("name", sorted(WRITTEN_BEFORE))
def test_reads_follow_the_wait(name):
    params, body = _kernel(name)
    waits = re.findall(r"wait_previous_kernel\(([^)]*)\)", body)
    assert len(waits) == 1
    named = {p.strip() for p in waits[0].split(",") if p.strip()}
    assert WRITTEN_BEFORE[name] <= named
    for p in named:
        decl = [d for d in params.split(",") if re.search(r"\b%s\s*$" % p, d.strip())]
        decl += re.findall(r"\n  (const \w+ \*%s) = " % p, body[:body.index("wait_previous_kernel")])  # or a copy of one
        assert len(decl) == 1 and "*" in decl[0] and "__restrict__" not in decl[0], p


def test_every_kernel_with_the_attribute_waits():
    for name in set(re.findall(r"launch_after\([^,]*,\s*(k_\w+)", SOURCE)):
        assert "wait_previous_kernel(" in _kernel(name)[1], name


def test_retry_phase_is_acquired_by_the_thread_that_reads_it():
    """The thread that saw the phase word change fences before the barrier that lets its block in (the word itself is
    polled relaxed), and so does each thread that counts a phase's last pieces before it reads what they wrote."""
    body = _kernel("k_retry")[1]
    enter = body[body.index("const auto enter"):]
    enter = enter[:enter.index("};")]
    assert enter.index("fence_gpu()") < enter.index("atomicAdd") < enter.index("current = to")
    last = body[body.index("+ held == n"):]
    assert last.index("__threadfence()") < last.index("__ldcg")
