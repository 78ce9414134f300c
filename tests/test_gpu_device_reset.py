"""A recount before and after the caller's cudaDeviceReset, which ends the process's own context: in a process of its own."""
import glob
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _runtime():
    for base in sys.path + ["/usr/local/cuda/lib64"]:
        for pattern in ("nvidia/cuda_runtime/lib/libcudart.so.*", "libcudart.so.*"):
            for found in glob.glob(os.path.join(base, pattern)):
                return found
    return None


def test_recount_works_across_a_device_reset(ccb, cuda_device):
    """The recount's scratch comes from a kept pool, which the reset takes away with the context; the next recount makes
    another.  Twice over, by popcount and by contraction."""
    runtime = _runtime()
    if runtime is None:
        pytest.skip("no shared CUDA runtime to reset the device with")
    run = subprocess.run([sys.executable, os.path.abspath(__file__), runtime], cwd=REPO, capture_output=True, text=True,
                         timeout=120)
    assert run.returncode == 0, run.stdout + run.stderr
    assert run.stdout.split() == ["equal"] * 3


def _child(runtime):
    import ctypes as C

    import numpy as np
    sys.path[:0] = [os.path.join(REPO, "oracle"), REPO]
    import cuda_graph_clustering_b200 as ccb
    from oracle import Oracle
    rt = C.CDLL(runtime)
    oracle = Oracle()

    def ok(status):
        assert status == 0, status

    def recount(n, k, count):
        bits, edges = oracle.erdos_renyi(n, 0.3, n)
        bits = np.ascontiguousarray(np.pad(bits, ((0, 0), (0, -bits.shape[1] % 4))))
        labels = np.random.default_rng(n).integers(0, k, (count, n)).astype(np.int32)
        f = np.zeros(count, np.int64)
        device = []
        for host in (bits, labels, f):
            p = C.c_void_p()
            ok(rt.cudaMalloc(C.byref(p), C.c_size_t(host.nbytes)))
            ok(rt.cudaMemcpy(p, host.ctypes.data_as(C.c_void_p), C.c_size_t(host.nbytes), 1))
            device.append(p.value)
        ccb.evaluate_labelings(device[0], n, bits.shape[1], edges, k, count, device[1], device[2])
        ok(rt.cudaMemcpy(f.ctypes.data_as(C.c_void_p), C.c_void_p(device[2]), C.c_size_t(f.nbytes), 2))
        assert f.tolist() == [oracle.rebuild(bits[:, :(n + 31) // 32].copy(), edges, k, row)[0] for row in labels]

    for turn in range(3):
        recount(700, 5, 3)
        recount(2000, 40, 9)
        ccb.lib().ccb_release_cache()
        recount(700, 5, 3)
        print("equal", flush=True)
        if turn < 2:
            ok(rt.cudaDeviceReset())


if __name__ == "__main__":
    _child(sys.argv[1])
