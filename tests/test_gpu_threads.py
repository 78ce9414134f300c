"""Calls from several host threads at once, each on its own stream."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_contractions_of_different_sizes_in_two_threads(ccb, oracle, cuda_device):
    """The contraction's shared memory depends on its columns (16 to 256 a CTA): the limit that one thread's call sets holds
    for the kernel, so a call of few columns must not lower it between another's set-up and its launch."""
    import torch
    n, k = 1000, 16
    bits, edges = oracle.erdos_renyi(n, 0.3, 5)
    wide = torch.from_numpy(np.ascontiguousarray(bits).view(np.int32)).cuda()  # 32 words a row: whole 16-byte groups
    rng = np.random.default_rng(1)
    jobs = []
    for count in (1, 600):
        labels = rng.integers(0, k, (count, n)).astype(np.int32)
        jobs.append((count, labels, torch.from_numpy(labels).cuda(), torch.empty(count, dtype=torch.int64, device="cuda"),
                     torch.cuda.Stream()))
    torch.cuda.synchronize()
    errors = []

    def repeat(count, _, labels, f, stream):
        try:
            for _ in range(1500):
                ccb.evaluate_labelings_tensor(wide.data_ptr(), n, wide.shape[1], edges, k, count, labels.data_ptr(),
                                              f.data_ptr(), stream=stream.cuda_stream)
        except Exception as e:  # noqa: BLE001 (reported by the test)
            errors.append(e)

    threads = [threading.Thread(target=repeat, args=job) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for count, labels, _, f, _ in jobs:
        want = [oracle.rebuild(bits, edges, k, row)[0] for row in labels[:3]]
        assert f[:3].tolist() == want


def test_solvers_made_in_two_threads(ccb, oracle, cuda_device):
    """Solvers of one kernel instance with different needs of shared memory, made and run at the same time."""
    cases = []
    for n in (1400, 6000):  # both windowed, k = 3, h in shared memory
        bits, edges = oracle.erdos_renyi(n, 0.3, n)
        cases.append((ccb.DeviceGraph(ccb.Graph(n, bits, edges)), ccb.PbilsParams(k=3, population=4, iterations=1, seed=n)))
    want = [ccb.Solver(g, p).pbils(p) for g, p in cases]
    errors = []

    def repeat(case, expected):
        try:
            for _ in range(30):
                solver = ccb.Solver(*case)
                got = solver.pbils(case[1])
                assert got.objective == expected.objective and np.array_equal(got.labels, expected.labels)
                solver.close()
        except Exception as e:  # noqa: BLE001 (reported by the test)
            errors.append(e)

    threads = [threading.Thread(target=repeat, args=a) for a in zip(cases, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
