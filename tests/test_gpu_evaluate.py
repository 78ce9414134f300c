"""Device recount (ccb_evaluate_labelings) against the CPU oracle's Rebuild and ObjectiveBitwise."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(ccb, torch, bits, edges, k, labels):
    count, n = labels.shape
    dbits = torch.from_numpy(bits.view(np.int32)).cuda()
    dlab = torch.from_numpy(labels).cuda()
    f = torch.empty(count, dtype=torch.int64, device="cuda")
    sizes = torch.empty((count, k), dtype=torch.int32, device="cuda")
    g = torch.empty((count, k, max(n, 1)), dtype=torch.int32, device="cuda")
    ccb.evaluate_labelings(dbits.data_ptr(), n, bits.shape[1], edges, k, count, dlab.data_ptr(), f.data_ptr(),
                           sizes.data_ptr(), g.data_ptr())
    torch.cuda.synchronize()
    return f.cpu().numpy(), sizes.cpu().numpy(), g.cpu().numpy()[:, :, :n]


@pytest.mark.parametrize("n,k", [(1, 1), (31, 2), (32, 3), (33, 5), (257, 7), (1000, 64), (3000, 9)])
def test_evaluate_matches_oracle(ccb, oracle, cuda_device, n, k):
    import torch
    rng = np.random.default_rng(n * 7 + k)
    bits, edges = oracle.erdos_renyi(n, 0.37, n + k)
    labels = rng.integers(0, k, (5, n)).astype(np.int32)
    f, sizes, g = _run(ccb, torch, bits, edges, k, labels)
    for i in range(labels.shape[0]):
        fo, go, so = oracle.rebuild(bits, edges, k, labels[i])
        assert f[i] == fo == oracle.objective_bitwise(bits, labels[i])
        assert np.array_equal(sizes[i], so) and np.array_equal(g[i], go)


def test_evaluate_flags_bad_labels(ccb, oracle, cuda_device):
    import torch
    bits, edges = oracle.erdos_renyi(100, 0.5, 1)
    labels = np.zeros((2, 100), np.int32)
    labels[1, 7] = 3
    f, _, _ = _run(ccb, torch, bits, edges, 3, labels)
    assert f[0] == oracle.objective_bitwise(bits, labels[0]) and f[1] == -1


def test_evaluate_recounts_a_solve(ccb, oracle, cuda_device):
    import torch
    bits, edges = oracle.erdos_renyi(2000, 0.3, 4)
    r = ccb.SolveGpu(ccb.Graph(2000, bits, edges), ccb.PbilsParams(k=6, population=32, iterations=5))
    f, _, _ = _run(ccb, torch, bits, edges, 6, r.labels.reshape(1, -1).astype(np.int32))
    assert f[0] == r.objective


# The tiles of the spread-out recount: rows past a block's and a warp's last, cluster chunks of 4, 8 and 16 and their
# remainders, one labeling and many, rows wider than ceil(n / 32) words, no optional outputs
@pytest.mark.parametrize("n,k,count,pad", [(127, 4, 1, 0), (129, 5, 3, 1), (64, 8, 2, 0), (65, 9, 1, 3), (2049, 16, 1, 0),
                                           (1023, 17, 2, 1), (33, 33, 70, 0), (4097, 3, 1, 2), (100, 1, 300, 0),
                                           (2000, 40, 9, 1), (2000, 40, 9, 0)])  # by contraction (64-word rows), by popcount
def test_evaluate_tiles_match_oracle(ccb, oracle, cuda_device, n, k, count, pad):
    import torch
    rng = np.random.default_rng(n + k)
    bits, edges = oracle.erdos_renyi(n, 0.3, n)
    wide = np.ascontiguousarray(np.pad(bits, ((0, 0), (0, pad))))
    labels = rng.integers(0, k, (count, n)).astype(np.int32)
    labels[-1, n // 2] = k if k % 2 else -1  # not a label: f = -1, the vertex in no cluster
    f, sizes, g = _run(ccb, torch, wide, edges, k, labels)
    for i in range(count - 1):
        fo, go, so = oracle.rebuild(bits, edges, k, labels[i])
        assert f[i] == fo and np.array_equal(sizes[i], so) and np.array_equal(g[i], go)
    assert f[-1] == -1 and sizes[-1].sum() == n - 1
    dbits, dlab = torch.from_numpy(wide.view(np.int32)).cuda(), torch.from_numpy(labels).cuda()
    alone = torch.empty(count, dtype=torch.int64, device="cuda")
    ccb.evaluate_labelings(dbits.data_ptr(), n, wide.shape[1], edges, k, count, dlab.data_ptr(), alone.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(alone.cpu().numpy(), f)
    ccb.lib().ccb_release_cache()
