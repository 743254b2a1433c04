"""Host <-> device copies through the staging lanes: what goes in comes out, at the sizes where the path changes."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def round_trip(engine, n, k, seed):
    rng = np.random.default_rng(seed)
    P = rng.random((n, k), dtype=np.float32)
    ids = rng.integers(0, n, (n, k), dtype=np.int32)
    with engine.Session(n, k) as s:
        s.set_affinities(P, ids)
        P2, ids2 = s.get_affinities()
    return np.array_equal(P, P2) and np.array_equal(ids, ids2)


# 4 n k bytes: just below and at the 24 MiB from which copies are staged, one value over (a last chunk of 4 bytes), a
# last chunk that is not full, and more chunks than the lanes have slots
@pytest.mark.parametrize("n,k", [(6 * MIB // 8 - 1, 8), (6 * MIB // 8, 8), (6 * MIB + 1, 1), (100003, 67), (700001, 16)])
def test_round_trip(engine, n, k):
    assert round_trip(engine, n, k, n)


def test_threads_share_the_kept_resources(engine):
    ok = []
    threads = [threading.Thread(target=lambda t=t: ok.append(round_trip(engine, 120000 + t, 55, t))) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert ok == [True] * 6
    engine.release_cached_memory()
    assert round_trip(engine, 120000, 55, 9)


RESET = """
import ctypes as C
import numpy as np
from tsne_cuda_b200 import _lib as e
cu = C.CDLL("libcuda.so.1")
rng = np.random.default_rng(0)
small = rng.normal(0, 1, (2000, 10)).astype(np.float32)
large = rng.normal(0, 1, (30000, 250)).astype(np.float32)     # staged copies, the blocked copy of P

def device(n):
    p = C.c_uint64()
    assert cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(n)) == 0
    return p

def search():
    n, d = small.shape
    x, i, q = device(small.nbytes), device(n * 20 * 4), device(n * 20 * 4)
    ids = np.empty((n, 20), np.int32)
    assert cu.cuMemcpyHtoD_v2(x, C.c_void_p(small.ctypes.data), C.c_size_t(small.nbytes)) == 0
    e.check(e.lib.b200tsne_knn_noalloc(C.c_void_p(x.value), n, d, 20, C.c_void_p(i.value), C.c_void_p(q.value), None))
    assert cu.cuMemcpyDtoH_v2(C.c_void_p(ids.ctypes.data), i, C.c_size_t(ids.nbytes)) == 0
    return ids

def everything():
    ids, _ = e.knn(small, 20)
    assert np.array_equal(ids, search())
    Y = [e.fit(x, num_neighbors=20, perplexity=6.0, iterations=70, random_seed=1)[0] for x in (small, large)]
    assert all(np.isfinite(y).all() for y in Y)
    return ids, e.knn(large, 20)[0]

a = everything()
left = e.Session(2000, 20)                                     # outlives its context
left.set_affinities(np.full((2000, 20), 1e-5, np.float32), a[0])
left.set_embedding(rng.normal(0, 1, (2, 2000)).astype(np.float32))
left.run(20)
for _ in range(2):
    assert cu.cuDevicePrimaryCtxReset_v2(0) == 0
    b = everything()
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
left.close()
b = everything()
assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
e.release_cached_memory()
"""


def test_calls_after_a_device_reset():
    """Resetting the device (as cudaDeviceReset does) ends the kept streams, events, pinned memory and executables with
    its context: the next call makes its own."""
    subprocess.run([sys.executable, "-c", RESET], check=True, cwd=ROOT, timeout=200)
