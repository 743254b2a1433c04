"""The search at its limits: norms beyond the range of floats (every key of a sample is infinite, and the padding of the
last tile must not pass), several threads at once, more rows than one batch of queries, and device memory."""
import ctypes as C
import threading

import numpy as np
import pytest

from conftest import mixture

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [20, 100])
def test_infinite_norms(engine, monkeypatch, d):
    X = mixture(2100, d, d)
    X[:2000] += np.float32(3e19)    # |x|^2 = inf for these, the others far below them
    a = engine.knn(X, 30)
    monkeypatch.setenv("B200TSNE_KNN", "simt")
    b = engine.knn(X, 30)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("widths", [(20, 46, 62), (9, 30, 63), (70, 500, 33)])
def test_threads_search_points_of_different_width(engine, widths):
    """The kernels' shared memory depends on the width: no thread's call may take from another's what it launches with."""
    X = [mixture(2300, d, d) for d in widths]
    want = [engine.knn(x, 30) for x in X]
    bad = []

    def search(i):
        for _ in range(400):
            try:
                ids, d2 = engine.knn(X[i], 30)
                if not (np.array_equal(ids, want[i][0]) and np.array_equal(d2, want[i][1])):
                    bad.append(widths[i])
            except engine.TsneError as e:
                bad.append(str(e))

    threads = [threading.Thread(target=search, args=(i % len(X),)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


BATCH = 1 << 20    # queries of one batch, and rows whose distances to the cells are kept


@pytest.mark.parametrize("n,q", [(BATCH, (0, 3)), (BATCH + 1, (0, 3)), (BATCH + 1, (BATCH - 2, BATCH + 1)), (BATCH + 70001, (BATCH, BATCH + 3))])
def test_around_one_batch(engine, oracle_cpu, n, q):
    """Clustered points (most tiles are skipped), lists of a few rows against the oracle: one query range alone, and out of
    the search of all rows, whose cells come from the kept distances up to the batch's size and from its own beyond."""
    X = mixture(n, 6, 5, k=40)
    ids_o, d2_o = oracle_cpu.knn(X, 9, q_lo=q[0], q_hi=q[1])
    ids, d2 = engine.knn(X, 9, q_lo=q[0], q_hi=q[1])
    assert np.array_equal(ids, ids_o) and np.array_equal(d2, d2_o)
    ids, d2 = engine.knn(X, 9)
    assert np.array_equal(ids[q[0]:q[1]], ids_o) and np.array_equal(d2[q[0]:q[1]], d2_o)


def _peak(engine, call):
    """Most device memory in use during `call` (the library takes all of it from the device's default pool)."""
    cu = C.CDLL("libcuda.so.1")
    engine.knn(mixture(300, 4, 1), 5)
    pool, used = C.c_void_p(), C.c_uint64(0)
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert cu.cuMemPoolSetAttribute(pool, 8, C.byref(used)) == 0            # CU_MEMPOOL_ATTR_USED_MEM_HIGH
    call()
    assert cu.cuMemPoolGetAttribute(pool, 8, C.byref(used)) == 0
    return used.value


def test_device_memory_per_row(engine):
    """A search holds, per database row of 4 dimensions and 8 neighbours of few queries: the row 16 bytes, its copy in
    visiting order 16, its operand image 32, its list entry 4, its cell and the distance to it 5.  Per row that is a query
    too: its lists 64, image 32, norms 16, list entries 12, threshold and counts 12, segments 4, 1,024 candidates 8,192, and
    its distances to the 64 cells 256, once.  (These were kept for every database row, and once more for the queries.)"""
    n = [1200000, 1700000]
    X = mixture(n[1], 4, 2, k=30)
    few = [_peak(engine, lambda: engine.knn(X[:m], 8, q_lo=0, q_hi=1000)) for m in n]
    assert (few[1] - few[0]) / (n[1] - n[0]) < 73 + 16
    n = [400000, 900000]
    every = [_peak(engine, lambda: engine.knn(X[:m], 8)) for m in n]
    assert (every[1] - every[0]) / (n[1] - n[0]) < 73 + 64 + 32 + 16 + 12 + 12 + 4 + 8192 + 256 + 64
