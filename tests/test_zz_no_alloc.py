"""GPU test of b200tsne_knn_noalloc, the neighbour search for hosts that may not allocate device memory
inside the call (their own pool owns the device, or the allocator's implicit synchronisation is not
acceptable): the caller hands in device buffers, the library's scratch is a fixed array in its image.

Collected last on purpose (file name): a stop-at-first-failure run has then exercised everything else."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, mixture

pytestmark = pytest.mark.gpu


def _search(engine, torch, X, K):
    """One call through the C ABI on caller-owned device buffers; returns host copies."""
    N, D = X.shape
    x_d = torch.from_numpy(X).cuda()
    ids_d = torch.empty((N, K), dtype=torch.int32, device="cuda")
    d2_d = torch.empty((N, K), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    rc = engine.lib.b200tsne_knn_noalloc(C.c_void_p(x_d.data_ptr()), N, D, K, C.c_void_p(ids_d.data_ptr()),
                                         C.c_void_p(d2_d.data_ptr()), None)
    assert rc == 0, engine.lib.b200tsne_last_error()
    torch.cuda.synchronize()   # the call only queues the work
    return ids_d.cpu().numpy(), d2_d.cpu().numpy()


def test_no_alloc_search_matches_allocating_search_twice(engine):
    torch = pytest.importorskip("torch")
    assert engine.lib.b200tsne_knn_noalloc_max_elements() == 4 << 20
    # two calls in a row with different shapes: the second must not see anything of the first in the scratch
    for n, d, k, seed in ((3000, 20, 15, 1), (1777, 33, 40, 2)):
        X = mixture(n, d, seed)
        ids, d2 = _search(engine, torch, X, k)
        ids_ref, d2_ref = engine.knn(X, k)          # the existing entry point (allocates its own scratch)
        assert np.array_equal(ids, ids_ref)          # integer output: bit-exact
        assert np.array_equal(d2, d2_ref)            # canonical fp32 distances: bit-exact as well


def test_no_alloc_search_rejects_oversized_input(engine):
    torch = pytest.importorskip("torch")
    limit = engine.lib.b200tsne_knn_noalloc_max_elements()
    buf = torch.zeros(16, device="cuda")
    n = limit // 8 + 1                               # n * 8 > limit: refused before anything is read
    rc = engine.lib.b200tsne_knn_noalloc(C.c_void_p(buf.data_ptr()), n, 8, 4, C.c_void_p(buf.data_ptr()),
                                         C.c_void_p(buf.data_ptr()), None)
    assert rc == -4 and b"exceeds the built-in scratch" in engine.lib.b200tsne_last_error()
    assert engine.lib.b200tsne_knn_noalloc(None, 10, 8, 4, None, None, None) == -1


def test_one_call_of_any_size_loads_what_later_ones_launch():
    """In a fresh process, after one small call: the first call of another size (other forms of the distance and selection
    kernels, the list search) takes the host no longer than later ones, and sizes never called before are captured and
    replayed on other points, lists as from the allocating search.  (A kernel still to be loaded costs the first call 20 to
    70 us beside 15 to 20: 3.6 times the later ones for the two sizes together; the bar leaves half of that for the host.)"""
    code = """
import ctypes as C
import time
import numpy as np, torch
from tsne_cuda_b200 import _lib as e
def buffers(n, d, k):
    return torch.zeros(n, d, device="cuda"), torch.zeros(n, k, dtype=torch.int32, device="cuda"), torch.zeros(n, k, device="cuda")
def call(b, st):
    (n, d), k = b[0].shape, b[1].shape[1]
    t = time.perf_counter()
    e.check(e.lib.b200tsne_knn_noalloc(b[0].data_ptr(), n, d, k, b[1].data_ptr(), b[2].data_ptr(), C.c_void_p(st.cuda_stream)))
    return time.perf_counter() - t
sizes = [(40, 3, 5), (4099, 64, 16), (8000, 7, 64), (12288, 5, 30), (3000, 9, 600), (12500, 7, 10)]
bufs = [buffers(*s) for s in sizes]
st = torch.cuda.Stream()
small = buffers(300, 4, 4)
for _ in range(3):
    call(small, st)
    st.synchronize()
first = later = 0.0
for s in ((1500, 20, 32), (13000, 7, 10)):
    b = buffers(*s)
    torch.cuda.synchronize()
    t = []
    for _ in range(8):
        t.append(call(b, st))
        st.synchronize()
    first += t[0]
    later += sorted(t[1:])[3]
assert first < 2.2 * later, (first, later)
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g, stream=st):
    for b in bufs: call(b, st)
rng = np.random.default_rng(0)
X = [rng.normal(0, 1, (n, d)).astype(np.float32) for n, d, k in sizes]
for b, x in zip(bufs, X): b[0].copy_(torch.from_numpy(x))
torch.cuda.synchronize()
g.replay()
torch.cuda.synchronize()
for b, x in zip(bufs, X):
    ids, d2 = e.knn(x, b[1].shape[1])
    assert np.array_equal(ids, b[1].cpu().numpy()) and np.array_equal(d2, b[2].cpu().numpy()), x.shape
"""
    subprocess.run([sys.executable, "-c", code], check=True, cwd=ROOT, timeout=200, env=dict(os.environ, CUDA_MODULE_LOADING="LAZY"))
