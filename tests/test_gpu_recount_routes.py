"""The recount by each of its routes: popcount, contraction, popcount after a contraction that gave up, inside a capture.

ccb_evaluate_labelings picks popcount or the contraction by size; ccb_evaluate_labelings_noalloc is always popcount and
ccb_evaluate_labelings_tensor always the contraction, so a comparison of the two really compares two computations."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(ccb, n, k, count, density, seed):
    import torch
    host = ccb.DeviceGraph.erdos_renyi(n, density, seed).download()
    words = host.bits.shape[1]
    padded = np.zeros((n, (words + 3) // 4 * 4), np.uint32)
    padded[:, :words] = host.bits
    labels = np.random.default_rng(seed).integers(0, k, (count, n)).astype(np.int32)
    return host, torch.from_numpy(padded.view(np.int32)).cuda(), labels, torch.from_numpy(labels).cuda()


def _outputs(n, k, count):
    import torch
    return (torch.full((count,), -7, dtype=torch.int64, device="cuda"),
            torch.full((count, k), -7, dtype=torch.int32, device="cuda"),
            torch.full((count, k, n), -7, dtype=torch.int32, device="cuda"))


def _call(fn, bits, n, edges, k, count, labels, out, stream=0):
    return fn(bits.data_ptr(), n, bits.shape[1], edges, k, count, labels.data_ptr(), *(o.data_ptr() for o in out), stream)


@pytest.mark.parametrize("n,k,count,density", [
    (2000, 64, 64, 0.4),    # 4096 columns
    (33000, 9, 20, 0.01),   # 180 columns, 129 row tiles of 256
    (65536, 2, 128, 0.02), (65536, 3, 128, 0.02)])
def test_contraction_equals_the_popcount_that_cannot_dispatch(ccb, oracle, cuda_device, n, k, count, density):
    import torch
    host, bits, labels, dlabels = _inputs(ccb, n, k, count, density, n + k)
    by = [_outputs(n, k, count) for _ in range(3)]
    for fn, out in zip((ccb.evaluate_labelings_noalloc, ccb.evaluate_labelings_tensor, ccb.evaluate_labelings), by):
        _call(fn, bits, n, host.edges, k, count, dlabels, out)
    torch.cuda.synchronize()
    for other in by[1:]:
        for a, b in zip(by[0], other):
            assert torch.equal(a, b)
    assert int(by[0][0][-1]) == oracle.objective_bitwise(host.bits, labels[-1])


@pytest.mark.parametrize("n,k,count", [(128, 2, 1), (129, 7, 3), (1000, 5, 129), (700, 64, 33), (2049, 16, 5)])
def test_labelings_are_counted_again_when_the_contraction_gave_up(ccb, oracle, cuda_device, n, k, count):
    """The wait is marked as given up from the start (no kernel waits): f is the objective or -1, never -2."""
    import torch
    host, bits, labels, dlabels = _inputs(ccb, n, k, count, 0.3, n)
    if count > 1:
        labels[-1, n // 2] = k  # not a label
        dlabels.copy_(torch.from_numpy(labels))
    again = ccb.lib().ccb_test_recount_gave_up
    again.restype = C.c_int
    again.argtypes = [C.c_void_p, C.c_uint32, C.c_uint32, C.c_uint64, C.c_int32, C.c_int32] + [C.c_void_p] * 5
    out = _outputs(n, k, count)
    assert _call(again, bits, n, host.edges, k, count, dlabels, out) == 0
    f = torch.full((count,), -7, dtype=torch.int64, device="cuda")
    assert again(bits.data_ptr(), n, bits.shape[1], host.edges, k, count, dlabels.data_ptr(), f.data_ptr(), None, None, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(f, out[0])
    f, sizes, g = (o.cpu().numpy() for o in out)
    for i in range(count):
        if count > 1 and i == count - 1:
            assert f[i] == -1 and sizes[i].sum() == n - 1
        else:
            fo, go, so = oracle.rebuild(host.bits, host.edges, k, labels[i])
            assert f[i] == fo and np.array_equal(sizes[i], so) and np.array_equal(g[i], go)


@pytest.mark.parametrize("n,k,count", [(1000, 5, 3), (2000, 40, 9)])  # by popcount, by contraction
def test_captured_recount(ccb, oracle, cuda_device, n, k, count):
    import torch
    host, bits, labels, dlabels = _inputs(ccb, n, k, count, 0.3, n)
    out = _outputs(n, k, count)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        _call(ccb.evaluate_labelings, bits, n, host.edges, k, count, dlabels, out, stream.cuda_stream)
    for turn in range(2):
        labels = (labels + turn) % k
        dlabels.copy_(torch.from_numpy(labels))
        graph.replay()
        torch.cuda.synchronize()
        for i in range(count):
            fo, go, so = oracle.rebuild(host.bits, host.edges, k, labels[i])
            assert int(out[0][i]) == fo
            assert np.array_equal(out[1][i].cpu().numpy(), so) and np.array_equal(out[2][i].cpu().numpy(), go)
