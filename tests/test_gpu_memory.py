"""Calls that run out of device memory: they fail alone, and what was there goes on working."""
import contextlib
import ctypes
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


@contextlib.contextmanager
def memory_left(mib):
    """All but about `mib` MiB of the device's free memory held by other buffers."""
    import torch
    held = []
    try:
        while True:
            spare = torch.cuda.mem_get_info()[0] - mib * MIB
            if spare < 4 * MIB:
                break
            held.append(torch.empty(spare // (2 * MIB) * (2 * MIB), dtype=torch.uint8, device="cuda"))
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


def _same(a, b):
    assert (a.objective, a.accepted_moves) == (b.objective, b.accepted_moves)
    assert np.array_equal(a.labels, b.labels)


def test_solver_survives_a_rebuild_kind_it_has_no_memory_for(ccb, cuda_device):
    """The popcount rebuild needs 17 MB of masks that a solver of the contraction never allocated."""
    graph = ccb.DeviceGraph.erdos_renyi(4100, 0.2, 3)
    p = ccb.PbilsParams(k=4, population=8192, iterations=1, early_stop=5, seed=2)
    solver = ccb.Solver(graph, p)
    assert "tcgen05" in solver.describe()
    want = solver.pbils(p)
    with memory_left(6):
        with pytest.raises(ccb.CcbError):
            solver.set_rebuild("popcount")
        assert "tcgen05" in solver.describe()
        _same(solver.pbils(p), want)
    solver.set_rebuild("popcount")
    assert "tcgen05" not in solver.describe()
    _same(solver.pbils(p), want)


def test_windows_that_do_not_fit_give_way(ccb, cuda_device):
    """n = 18000, k = 3: the streamed descent has its state in shared memory, the windowed one 108 KB a slot in L2.  With
    room for the one and not for the other a solver, and a one-call solve, take the first, with the same result."""
    p = ccb.PbilsParams(k=3, population=2048, iterations=1, early_stop=5, seed=2)
    graph = ccb.DeviceGraph.erdos_renyi(18000, 0.1, 3)
    host = graph.download()
    solver = ccb.Solver(graph, p)
    assert solver.describe().startswith("windowed")
    want = solver.pbils(p)
    solver.close()
    ccb.lib().ccb_release_cache()
    with memory_left(460):
        solver = ccb.Solver(graph, p)
        assert not solver.describe().startswith("windowed"), solver.describe()
        _same(solver.pbils(p), want)
        solver.close()
        for _ in range(2):
            _same(ccb.SolveGpu(host, p), want)
        ccb.lib().ccb_release_cache()
    solver = ccb.Solver(graph, p)
    assert solver.describe().startswith("windowed")
    solver.close()


def test_reported_memory_counts_what_is_allocated(ccb, cuda_device, capfd):
    """The masks of the popcount rebuild (17.3 MB here) are counted once they are there."""
    graph = ccb.DeviceGraph.erdos_renyi(4100, 0.2, 3)
    p = ccb.PbilsParams(k=4, population=8192, iterations=0, verbose=True)
    solver = ccb.Solver(graph, p)
    shown = []
    for kind in ("auto", "popcount"):
        solver.set_rebuild(kind)
        solver.pbils(p)
        ctypes.CDLL(None).fflush(None)
        shown.append(int(re.search(r"device memory: (\d+) MiB", capfd.readouterr().out).group(1)))
    assert 16 <= shown[1] - shown[0] <= 18, shown
