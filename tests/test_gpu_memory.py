"""Calls that run out of device memory: they fail alone, and what was there goes on working."""
import contextlib

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
