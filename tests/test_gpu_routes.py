"""One case and more of each descent that the windowed one did not replace, with the name of the kernel that runs: sparse
graphs below the line of the windows' rule, complete ones above it, batched instances of both engines.

Small instances follow the CPU oracle; larger ones the generic kernels of the same library, which the oracle pins at small
sizes (tests/test_gpu_parity.py)."""
import numpy as np
import pytest

from oracle import make_params

pytestmark = pytest.mark.gpu


def _same(got, want):
    assert (got.objective, got.iterations_done, got.accepted_moves, got.clusters_used) == \
        (want.objective, want.iterations_done, want.accepted_moves, want.clusters_used)
    assert np.array_equal(got.labels, want.labels)


@pytest.mark.parametrize("n,k,density,kernel", [
    (1400, 3, 0.0003, "packed k <= 8, registers,"), (2900, 4, 0.0003, "packed k <= 8, registers,"),
    (4090, 2, 0.0002, "packed k <= 8, registers,"),
    (4500, 2, 0.0005, "packed k <= 8, streamed from shared memory"), (9000, 3, 0.001, "packed k <= 8, streamed from shared memory"),
    (5000, 8, 0.001, "packed k <= 8, streamed from shared memory"),
    (13000, 6, 0.0005, "packed k <= 8, streamed from shared memory"),
    (20000, 5, 0.0004, "packed k <= 8, state in the distributed shared memory"),
    (17000, 8, 0.0004, "packed k <= 8, state in the distributed shared memory"),
    (1500, 12, 0.0004, "incremental 9 <= k <= 64, cached keys in registers, counters in shared memory"),
    (3000, 35, 0.01, "incremental 9 <= k <= 64, cached keys in registers, counters in shared memory"),
    (4000, 64, 0.01, "incremental 9 <= k <= 64, cached keys in registers, counters in L2"),
    (6000, 20, 0.001, "incremental 9 <= k <= 64, cached keys in registers, counters in L2"),
    (12000, 9, 0.0005, "incremental 9 <= k <= 64, cached keys in registers, counters in L2"),
    (17000, 10, 0.0005, "incremental 9 <= k <= 64, L2")])
def test_sparse_graphs_match_oracle(ccb, oracle, cuda_device, n, k, density, kernel):
    bits, edges = oracle.erdos_renyi(n, density, n + k)
    p = dict(k=k, population=3, iterations=2 if n < 5000 else 1, early_stop=10, gww=0.34, seed=5)
    solver = ccb.Solver(ccb.DeviceGraph(ccb.Graph(n, bits, edges)), ccb.PbilsParams(**p))
    assert solver.describe().startswith(kernel), solver.describe()
    _same(solver.pbils(ccb.PbilsParams(**p)), oracle.pbils(bits, edges, make_params(**p)))


def _against(ccb, n, k, density, pop, kernel, other, seed=3):
    graph = ccb.DeviceGraph.erdos_renyi(n, density, n + k)
    p = dict(k=k, population=pop, iterations=1, early_stop=10, seed=seed)
    solver = ccb.Solver(graph, ccb.PbilsParams(**p))
    assert solver.describe().startswith(kernel), solver.describe()
    q = ccb.PbilsParams(**p, ls_kernel=other)
    _same(solver.pbils(ccb.PbilsParams(**p)), ccb.Solver(graph, q).pbils(q))


# the streamed state in L2: more clusters of CTAs than run at once; with L2 priorities where it takes over 3/8 of L2
@pytest.mark.parametrize("n,k,density,pop,kernel", [
    (20000, 5, 0.0004, 80, "packed k <= 8, streamed from L2,"),
    (26000, 8, 0.0004, 120, "packed k <= 8, streamed from L2 (state evict_last, rows evict_first)")])
def test_sparse_graphs_in_l2_match_the_generic_kernel(ccb, cuda_device, n, k, density, pop, kernel):
    _against(ccb, n, k, density, pop, kernel, ccb.LS_GLOBAL)


# the wide forms: dense ones of k = 2 and 3 (average degree above n / 8, gains narrow because the graph is nearly complete),
# degree-proportional ones, the incremental one
@pytest.mark.parametrize("n,k,density,kernel", [
    (33000, 2, 0.99, "packed wide k = 2 (e = G1 - G0 and the label"),
    (33001, 3, 0.999, "packed wide k = 3 (three 20-bit counters"),
    (33000, 2, 0.004, "packed wide k = 2, degree-proportional (per-thread best of each cluster), int16 state in shared memory"),
    (33001, 3, 0.001, "packed wide k = 3, degree-proportional (per-thread best of each (cluster, target) class), 26-bit records"),
    (33000, 5, 0.0002, "incremental wide"), (32801, 40, 0.001, "incremental wide")])
def test_wide_forms_match_the_generic_kernel(ccb, cuda_device, n, k, density, kernel):
    _against(ccb, n, k, density, 2, kernel, ccb.LS_WIDE)


# the windowed wide form to the largest n, a bound of each way in which the moves are made
@pytest.mark.parametrize("n,k,density", [(65536, 2, 0.1), (65536, 4, 0.02), (65535, 8, 0.02), (45000, 14, 0.02), (45001, 20, 0.02)])
def test_windowed_wide_form_at_large_sizes(ccb, cuda_device, n, k, density):
    _against(ccb, n, k, density, 1, "windowed wide", ccb.LS_WIDE)


SPARSE = [(1400, 3, 0.0003), (2900, 12, 0.0005), (3000, 40, 0.01), (4500, 5, 0.0005), (17000, 10, 0.0005), (9000, 9, 0.0005),
          (300, 4, 0.05)]
LARGE = [(16384, 2, 0.2), (16500, 5, 0.2), (16400, 8, 0.1), (17001, 14, 0.1), (16500, 40, 0.2)]  # windowed, counters not in 15 bits


@pytest.mark.parametrize("engine", ["lockstep", "flow"])
@pytest.mark.parametrize("mix", [SPARSE, LARGE], ids=["sparse", "large"])
def test_batches_match_the_plain_solve(ccb, cuda_device, engine, mix):
    batch = ccb.Batch(engine=engine)
    runs = []
    for i, (n, k, density) in enumerate(mix):
        graph = ccb.DeviceGraph.erdos_renyi(n, density, 70 + i)
        p = ccb.PbilsParams(k=k, population=5, iterations=2, early_stop=10, seed=i)
        assert ccb.Solver(graph, p).describe().startswith("windowed") == (mix is LARGE)
        runs.append((batch.add(graph, p), graph, p))
    batch.run()
    for i, graph, p in runs:
        _same(batch.result(i), ccb.Solver(graph, p).pbils(p))
    batch.close()


@pytest.mark.parametrize("threads", [256, 512, 1024])
def test_tuned_batch_of_sparse_graphs_takes_the_global_form(ccb, cuda_device, threads):
    """use_kind 2 still applies to instances that run the incremental descent with its state in L2."""
    before = ccb.get_tuning()
    ccb.set_tuning([dict(kind=-1, n_min=0, n_max=1 << 20, k_min=9, k_max=64, use_kind=2, threads=threads, blocks_per_sm=0,
                         max_slots=0)])
    try:
        batch = ccb.Batch()
        runs = []
        for i, (n, k, density) in enumerate([(6000, 20, 0.001), (4000, 64, 0.01), (17000, 10, 0.0005)]):
            graph = ccb.DeviceGraph.erdos_renyi(n, density, 90 + i)
            p = ccb.PbilsParams(k=k, population=4, iterations=2, early_stop=10, seed=i)
            runs.append((batch.add(graph, p), graph, p))
        batch.run()
        assert f"incremental k=0 threads={threads}" in batch.describe(), batch.describe()
        for i, graph, p in runs:
            _same(batch.result(i), ccb.Solver(graph, p).pbils(p))
    finally:
        ccb.set_tuning(before)


@pytest.mark.parametrize("engine", ["lockstep", "flow"])
@pytest.mark.parametrize("n,k", [(14450, 8), (28910, 3)])
def test_batched_stream_at_the_edge_of_shared_memory(ccb, cuda_device, engine, n, k):
    """A streamed state of 226 KB fits beside the plain kernel's static shared memory, not beside the flow kernel's: the
    batch streams it from L2."""
    graph = ccb.DeviceGraph.erdos_renyi(n, 0.0004, 7)
    p = ccb.PbilsParams(k=k, population=3, iterations=1, early_stop=5, seed=2)
    plain = ccb.Solver(graph, p)
    assert plain.describe().startswith("packed k <= 8, streamed from shared memory")
    batch = ccb.Batch(engine=engine)
    i = batch.add(graph, p)
    batch.run()
    assert "stream k=%d threads=1024 vpt=4 smem=0" % k in batch.describe(), batch.describe()
    _same(batch.result(i), plain.pbils(p))
    batch.close()
