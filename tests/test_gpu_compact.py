"""The compact-pair register descent (csrc/ccb_descent_registers.cuh, k <= 8, n <= 1023) against the oracle: odd n (a pair
with one vertex), the edges of its thread shapes (256, 512, 1023 vertices) and of the 32-vertex row words, every k,
empty and complete graphs, whose gains all tie."""
import numpy as np
import pytest

from oracle import make_params

pytestmark = pytest.mark.gpu


def _check(ccb, oracle, bits, edges, **p):
    want = oracle.pbils(bits, edges, make_params(**p))
    got = ccb.SolveGpu(ccb.Graph(bits.shape[0], bits, edges), ccb.PbilsParams(**p))
    assert (got.objective, got.iterations_done, got.accepted_moves, got.clusters_used) == \
        (want.objective, want.iterations_done, want.accepted_moves, want.clusters_used)
    assert np.array_equal(got.labels, want.labels)


@pytest.mark.parametrize("n,k", [(2, 2), (3, 8), (31, 3), (32, 4), (33, 5), (127, 6), (128, 7), (129, 8), (255, 2),
                                 (256, 3), (257, 4), (511, 5), (512, 6), (513, 7), (1021, 8), (1022, 2), (1023, 3),
                                 (1023, 8), (1024, 4)])
def test_matches_oracle(ccb, oracle, cuda_device, n, k):
    bits, edges = oracle.erdos_renyi(n, 0.35, n + k)
    _check(ccb, oracle, bits, edges, k=k, population=6, iterations=4, early_stop=10, gww=0.25, seed=n)


@pytest.mark.parametrize("density", [0.0, 1.0])
@pytest.mark.parametrize("n,k", [(75, 8), (301, 3), (1023, 5)])
def test_gains_that_tie(ccb, oracle, cuda_device, n, k, density):
    bits, edges = oracle.erdos_renyi(n, density, 1)
    _check(ccb, oracle, bits, edges, k=k, population=4, iterations=2, early_stop=10, seed=9)
