"""The search at its limits: norms beyond the range of floats (every key of a sample is infinite, and the padding of the
last tile must not pass), and several threads at once."""
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
