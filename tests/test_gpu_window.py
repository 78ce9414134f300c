"""The windowed descent (csrc/ccb_descent_window.cuh) against the oracle: the edges of its 128-vertex quads and of the
sizes that select it, every compiled cluster bound, counters in shared memory and in L2, gains that tie by the
thousand, and the change between descents in the one-call cache."""
import numpy as np
import pytest

from oracle import make_params

pytestmark = pytest.mark.gpu


def _solve(ccb, oracle, bits, edges, **p):
    want = oracle.pbils(bits, edges, make_params(**p))
    got = ccb.SolveGpu(ccb.Graph(bits.shape[0], bits, edges), ccb.PbilsParams(**p))
    assert got.objective == want.objective
    assert np.array_equal(got.labels, want.labels)
    assert (got.iterations_done, got.accepted_moves, got.clusters_used) == \
        (want.iterations_done, want.accepted_moves, want.clusters_used)


def _plan(ccb, bits, edges, **p):
    graph = ccb.DeviceGraph(ccb.Graph(bits.shape[0], bits, edges))
    return ccb.Solver(graph, ccb.PbilsParams(**p)).describe()


# n around multiples of 128 (a quad), both sides of the smallest n of the k <= 8 form, members fewer than their slots (n < 1024),
# counters in shared memory and in L2 (k n large)
@pytest.mark.parametrize("n,k,density", [
    (1281, 2, 0.3), (1314, 8, 0.3), (1315, 2, 0.3), (1408, 3, 0.5), (1409, 4, 0.2), (1535, 5, 0.4), (1537, 6, 0.3), (2047, 7, 0.3), (2049, 8, 0.6),
    (33, 9, 0.5), (128, 16, 0.4), (127, 17, 0.4), (129, 32, 0.3), (300, 33, 0.3), (64, 64, 0.5), (1025, 9, 0.2),
    (2500, 16, 0.3), (1100, 32, 0.4), (1300, 64, 0.5), (9000, 13, 0.1), (12000, 8, 0.05),
    (16383, 3, 0.3), (16384, 2, 0.3)])  # the largest n whose h fit 15 bits, and the first past it
def test_matches_oracle(ccb, oracle, cuda_device, n, k, density):
    bits, edges = oracle.erdos_renyi(n, density, n + k)
    p = dict(k=k, population=4, iterations=3 if n < 3000 else 1, early_stop=10, gww=0.25, seed=n)
    # k <= 8 keeps the register descent while the bitset fits in shared memory (227 KB less 1 KB)
    assert _plan(ccb, bits, edges, **p).startswith("windowed") == (k > 8 or n * 16 * ((n + 127) // 128) > 231424)
    _solve(ccb, oracle, bits, edges, **p)


# Noise-free communities: whole communities tie, more vertices at the best gain than a window holds
@pytest.mark.parametrize("n,parts,k", [(3000, 2, 2), (2600, 3, 5), (2400, 2, 12), (1500, 4, 40)])
def test_gains_that_tie(ccb, oracle, cuda_device, n, parts, k):
    bits, edges, _ = oracle.planted(n, parts, False, 1.0, 0.0, 0.0, 3)
    p = dict(k=k, population=3, iterations=2, early_stop=10, seed=7)
    assert _plan(ccb, bits, edges, **p).startswith("windowed")
    _solve(ccb, oracle, bits, edges, **p)


def test_one_call_cache_follows_the_density(ccb, oracle, cuda_device):
    """A dense graph takes the windowed descent, an empty one of the same size does not; each call of an alternating
    sequence equals the oracle."""
    n = 1600
    dense = oracle.erdos_renyi(n, 0.4, 1)
    empty = (np.zeros_like(dense[0]), 0)
    p = dict(k=3, population=4, iterations=2, early_stop=10, seed=3)
    assert _plan(ccb, *dense, **p).startswith("windowed") and not _plan(ccb, *empty, **p).startswith("windowed")
    for bits, edges in (dense, empty, dense):
        _solve(ccb, oracle, bits, edges, **p)


# The wide form (32767 < n <= 65536, int32 population) against the generic wide kernel on the same graph: first and
# ragged sizes, the member caps of k <= 4, k <= 8 and larger k, every way the moves are made
@pytest.mark.parametrize("n,k,density", [(32768, 4, 0.02), (32897, 3, 0.05), (33003, 2, 0.3), (32769, 7, 0.05),
                                         (32800, 9, 0.05), (32770, 20, 0.1), (32900, 40, 0.2)])
def test_wide_matches_the_generic_kernel(ccb, cuda_device, n, k, density):
    graph = ccb.DeviceGraph.erdos_renyi(n, density, n + k)
    p = dict(k=k, population=3, iterations=1, early_stop=10, seed=n)
    auto = ccb.Solver(graph, ccb.PbilsParams(**p))
    assert auto.describe().startswith("windowed wide")
    got = auto.pbils(ccb.PbilsParams(**p))
    want = ccb.Solver(graph, ccb.PbilsParams(**p, ls_kernel=ccb.LS_WIDE)).pbils(
        ccb.PbilsParams(**p, ls_kernel=ccb.LS_WIDE))
    assert (got.objective, got.accepted_moves) == (want.objective, want.accepted_moves)
    assert np.array_equal(got.labels, want.labels)
