"""Which instances the windowed descent takes, and that it holds up where it could lose.

Vertices whose gains tie by the thousand: a window of them makes as many moves as any other."""
import numpy as np
import pytest

from oracle import make_params

pytestmark = pytest.mark.gpu


def _clock(ccb, solver, params):
    """ns of descent a move, the better of three solves."""
    solver.set_profiling(True)
    best = None
    for _ in range(3):
        r = solver.pbils(params)
        ns = solver.stats().descent_ms * 1e6 / max(r.accepted_moves, 1)
        best = ns if best is None else min(best, ns)
    return best


# Two communities of more vertices than a window holds (1024), every gain of a community the same.  With one move a window
# a move took 7.2 times as long as on the same communities with one pair in a thousand flipped, whose gains differ.
@pytest.mark.parametrize("n,parts,k", [(6000, 2, 2), (5000, 2, 3)])
def test_ties_cost_no_window_a_move(ccb, cuda_device, n, parts, k):
    p = ccb.PbilsParams(k=k, population=64, iterations=2, early_stop=10, seed=3)
    ns = []
    for flip in (0.0, 0.001):
        graph, _ = ccb.DeviceGraph.planted(n, parts, 1.0, 0.0, flip, 11)
        solver = ccb.Solver(graph, p)
        assert solver.describe().startswith("windowed")
        ns.append(_clock(ccb, solver, p))
    assert ns[0] < 4 * ns[1], ns


# The same ties against the oracle: closed twins (gains fall together), open twins (they rise), classes of both, with windows
# of vertex-keyed members (k <= 8), of members in order (k > 8) and of counters in shared memory (k > 32)
@pytest.mark.parametrize("n,parts,k,p_in,p_out", [
    (4000, 2, 3, 1.0, 0.0), (5000, 3, 4, 1.0, 0.0), (4100, 2, 16, 1.0, 0.0), (4200, 2, 40, 1.0, 0.0),
    (4800, 4, 3, 0.0, 1.0), (5000, 3, 4, 0.0, 1.0), (4100, 2, 16, 0.0, 1.0), (4800, 4, 40, 0.0, 1.0)])
def test_ties_match_oracle(ccb, oracle, cuda_device, n, parts, k, p_in, p_out):
    bits, edges, _ = oracle.planted(n, parts, False, p_in, p_out, 0.0, 5)
    p = dict(k=k, population=2, iterations=2, early_stop=10, seed=2)
    want = oracle.pbils(bits, edges, make_params(**p))
    solver = ccb.Solver(ccb.DeviceGraph(ccb.Graph(n, bits, edges)), ccb.PbilsParams(**p))
    assert solver.describe().startswith("windowed")
    got = solver.pbils(ccb.PbilsParams(**p))
    assert (got.objective, got.accepted_moves) == (want.objective, want.accepted_moves)
    assert np.array_equal(got.labels, want.labels)


# Populations that fill the SMs more than once, where other descents keep several slots on an SM: the route follows the load
# (n <= 2048, k <= 5 and n <= 1024, k > 8), and both sides of each line follow the oracle
@pytest.mark.parametrize("n,k,pop,density,windowed", [
    (1400, 2, 160, 0.5, True), (1400, 2, 240, 0.5, False), (1400, 3, 240, 0.5, False), (1400, 4, 300, 0.5, True),
    (1400, 5, 300, 0.1, False), (1400, 6, 300, 0.1, True),
    (200, 9, 148, 0.3, True), (200, 9, 150, 0.3, False), (460, 12, 150, 0.3, True), (460, 16, 150, 0.3, False),
    (560, 16, 150, 0.3, True), (560, 17, 150, 0.3, False), (900, 64, 150, 0.3, True), (850, 64, 150, 0.3, False),
    (1400, 60, 8, 0.3, False)])
def test_route_follows_the_load(ccb, oracle, cuda_device, n, k, pop, density, windowed):
    bits, edges = oracle.erdos_renyi(n, density, n + k)
    p = dict(k=k, population=pop, iterations=1, early_stop=10, seed=4)
    solver = ccb.Solver(ccb.DeviceGraph(ccb.Graph(n, bits, edges)), ccb.PbilsParams(**p))
    assert solver.describe().startswith("windowed") == windowed, solver.describe()
    got = solver.pbils(ccb.PbilsParams(**p))
    want = oracle.pbils(bits, edges, make_params(**p))
    assert (got.objective, got.accepted_moves) == (want.objective, want.accepted_moves)
    assert np.array_equal(got.labels, want.labels)
    one = ccb.SolveGpu(ccb.Graph(n, bits, edges), ccb.PbilsParams(**p))
    assert one.objective == want.objective and np.array_equal(one.labels, want.labels)


@pytest.mark.parametrize("engine,count,windowed", [("lockstep", 2, True), ("lockstep", 6, False), ("flow", 6, True)])
def test_batched_route_follows_the_load(ccb, cuda_device, engine, count, windowed):
    batch = ccb.Batch(engine=engine)
    p = [ccb.PbilsParams(k=20, population=60, iterations=3, early_stop=10, seed=s) for s in range(count)]
    graphs = [ccb.DeviceGraph.erdos_renyi(300, 0.3, 50 + i) for i in range(count)]
    ids = [batch.add(g, q) for g, q in zip(graphs, p)]
    batch.run()
    assert batch.describe().startswith("windowed") == windowed, batch.describe()
    for i, g, q in zip(ids, graphs, p):
        got, want = batch.result(i), ccb.Solver(g, q).pbils(q)
        assert (got.objective, got.accepted_moves) == (want.objective, want.accepted_moves)
        assert np.array_equal(got.labels, want.labels)
    batch.close()


# Open twins: the vertices of one part of a nearly complete multipartite graph.  Two large parts lose by windows (moves raise
# the gains of the twins), many parts and closed twins (communities) do not; the one-call cache follows.
@pytest.mark.parametrize("n,parts,k,p_in,p_out,flip,windowed", [
    (3000, 2, 3, 0.0, 1.0, 0.0, False), (3001, 2, 5, 0.0, 1.0, 0.0005, False), (3000, 2, 12, 0.0, 1.0, 0.0, True),
    (6000, 3, 2, 0.0, 1.0, 0.0, False), (6000, 3, 3, 0.0, 1.0, 0.0, True), (3000, 2, 3, 0.0, 1.0, 0.05, True),
    (3000, 8, 2, 0.0, 1.0, 0.0, True), (6000, 3, 2, 0.0, 1.0, 0.0005, True), (3000, 2, 3, 1.0, 0.0, 0.0, True), (36000, 2, 3, 0.0, 1.0, 0.0, False),
    (36000, 2, 4, 0.0, 1.0, 0.0, True)])
def test_open_twins_keep_the_other_descents(ccb, oracle, cuda_device, n, parts, k, p_in, p_out, flip, windowed):
    graph, _ = ccb.DeviceGraph.planted(n, parts, p_in, p_out, flip, 6)
    p = dict(k=k, population=2, iterations=1, early_stop=10, seed=2)
    solver = ccb.Solver(graph, ccb.PbilsParams(**p))
    assert solver.describe().startswith("windowed") == windowed, solver.describe()
    host = graph.download()
    want = oracle.pbils(host.bits, host.edges, make_params(**p)) if n < 10000 else \
        ccb.SolveGpu(host, ccb.PbilsParams(**p, ls_kernel=ccb.LS_WIDE))
    for got in (solver.pbils(ccb.PbilsParams(**p)), ccb.SolveGpu(host, ccb.PbilsParams(**p))):
        assert (got.objective, got.accepted_moves) == (want.objective, want.accepted_moves)
        assert np.array_equal(got.labels, want.labels)


def test_one_call_cache_follows_the_ties(ccb, oracle, cuda_device):
    p = dict(k=3, population=2, iterations=1, early_stop=10, seed=3)
    for p_in, p_out in ((0.0, 1.0), (0.6, 0.2), (0.0, 1.0)):
        bits, edges, _ = oracle.planted(2500, 2, True, p_in, p_out, 0.0, 3)
        want = oracle.pbils(bits, edges, make_params(**p))
        got = ccb.SolveGpu(ccb.Graph(2500, bits, edges), ccb.PbilsParams(**p))
        assert (got.objective, got.accepted_moves) == (want.objective, want.accepted_moves)
        assert np.array_equal(got.labels, want.labels)


# An edge count other than the bitset's shifts every objective by the difference and nothing else, also past 32 bits
@pytest.mark.parametrize("n,k", [(300, 4), (1023, 8), (1100, 3), (1500, 3), (700, 12)])
def test_edge_count_beyond_32_bits(ccb, oracle, cuda_device, n, k):
    bits, edges = oracle.erdos_renyi(n, 0.3, n)
    p = dict(k=k, population=4, iterations=2, early_stop=10, seed=3)
    want = oracle.pbils(bits, edges, make_params(**p))
    got = ccb.SolveGpu(ccb.Graph(n, bits, edges + (3 << 30)), ccb.PbilsParams(**p))
    assert (got.objective - (3 << 30), got.accepted_moves) == (want.objective, want.accepted_moves)
    assert np.array_equal(got.labels, want.labels)


# Sparse graphs, whose gains are few: the other side of the width line against each descent that the windows replaced
@pytest.mark.parametrize("n,k,density,windowed", [
    (1400, 2, 0.2, True), (1400, 2, 0.05, False), (2048, 8, 0.05, True), (2048, 8, 0.01, False),
    (2049, 2, 0.05, True), (2049, 2, 0.005, False), (4096, 8, 0.01, True), (4096, 8, 0.004, False),
    (4097, 2, 0.004, True), (4200, 2, 0.0015, False), (4200, 3, 0.0022, True), (9000, 3, 0.0028, True), (9000, 3, 0.002, False),
    (2000, 32, 0.0045, True), (2000, 32, 0.0022, False), (3001, 32, 0.0027, True)])
def test_route_follows_the_width_of_the_gains(ccb, oracle, cuda_device, n, k, density, windowed):
    bits, edges = oracle.erdos_renyi(n, density, n + k)
    p = dict(k=k, population=2, iterations=1, early_stop=10, seed=4)
    solver = ccb.Solver(ccb.DeviceGraph(ccb.Graph(n, bits, edges)), ccb.PbilsParams(**p))
    assert solver.describe().startswith("windowed") == windowed, solver.describe()
    got = solver.pbils(ccb.PbilsParams(**p))
    want = oracle.pbils(bits, edges, make_params(**p))
    assert (got.objective, got.accepted_moves) == (want.objective, want.accepted_moves)
    assert np.array_equal(got.labels, want.labels)
