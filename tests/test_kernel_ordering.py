"""Ordering that no result on one machine can show missing, looked for in the kernel sources (CPU only).

A warp's rescans read counters that other lanes of the warp have just stored: votes and shuffles in between order no
memory, so a __syncwarp() has to stand between the last store of a fold and the first vote that leads to a rescan.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda_graph_clustering_b200", "csrc")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


# file, function, the fold's last store of a counter, the rescan
FOLDS = [
    ("ccb_descent_window.cuh", "WindowMovesN", r"mem\.g\[to \* kLd \+ i\] =", r"WindowRescan\("),
    ("ccb_descent_incremental.cuh", "DescentIncremental", r"st\.g\[static_cast<size_t>\(to\) \* ld \+ u\] =",
     r"WarpRescan2\("),
    ("ccb_descent_incremental.cuh", "DescentIncrementalRegs", r"\bg\[static_cast<size_t>\(to\) \* ld \+ u\] =",
     r"WarpRescan2\("),
]


@pytest.mark.parametrize("name,function,store,rescan", FOLDS, ids=[f[1] for f in FOLDS])
def test_warp_is_synchronised_between_the_fold_and_the_rescans(name, function, store, rescan):
    text = source(name)
    body = text[re.search(r"void " + function + r"\(", text).start():]
    between = body[re.search(store, body).end():]
    between = between[:re.search(rescan, between).start()]
    vote = re.search(r"__ballot_sync\(", between)
    assert vote is not None
    assert "__syncwarp();" in between[:vote.start()]


def test_tensor_memory_loads_wait_in_their_own_statement():
    """A tcgen05.ld writes its registers after it was issued: the wait belongs to the same statement, so that nothing
    that reads them can come in between."""
    statements = re.findall(r"asm volatile\((.*?)\);", source("ccb_rebuild_tensor.cu"), flags=re.S)
    loads = [s for s in statements if "tcgen05.ld." in s]
    assert loads and all("tcgen05.wait::ld" in s for s in loads)


def test_a_rebuild_past_a_stop_touches_nothing():
    """The launches of a rebuild that were enqueued before the stop flag was seen run after it: whatever writes to the
    population is a kernel that looks at the flag, not a memset, which cannot."""
    text = source("ccb_rebuild_tensor.cu")
    body = text[text.index("cudaError_t LaunchLabelsZ("):]
    body = body[:body.index("\n}")]
    assert "k_labels_z" in body and "cudaMemset" not in body
    assert text.count("RebuildStopped(a)") >= 2
