"""Scans whose database tiles several blocks divide (few query blocks on many SMs): the blocks append to the same candidate
buffers.  The lists are defined operation by operation, so they equal the SIMT search's bit for bit."""
import numpy as np
import pytest

from conftest import mixture

pytestmark = pytest.mark.gpu


def both(engine, monkeypatch, X, k, **ranges):
    a = engine.knn(X, k, **ranges)
    st = engine.knn_last_stats()
    assert st["tensor_core"] == 1
    monkeypatch.setenv("B200TSNE_KNN", "simt")
    b = engine.knn(X, k, **ranges)
    assert engine.knn_last_stats()["tensor_core"] == 0
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    return st


# one block of queries and up to sixteen; narrow and wide points; the last unit, tile and chunk partly filled
@pytest.mark.parametrize("n,d,k", [(2048, 7, 5), (2049, 63, 90), (2177, 64, 64), (4095, 30, 150), (5003, 257, 224), (9001, 784, 90)])
def test_few_query_blocks(engine, monkeypatch, n, d, k):
    from tsne_cuda_b200 import datasets
    X = datasets.mnist_shaped(n, d, seed=n) if d == 784 else mixture(n, d, n + d)
    st = both(engine, monkeypatch, X, k)
    assert st["rows_recomputed"] <= 0.02 * n


@pytest.mark.parametrize("d", [20, 100])
@pytest.mark.parametrize("q_lo,q_hi,db_lo,db_hi", [(0, 1, 0, 30000), (777, 906, 5, 29990), (0, 700, 15000, 30000)])
def test_short_query_ranges(engine, monkeypatch, d, q_lo, q_hi, db_lo, db_hi):
    both(engine, monkeypatch, mixture(30000, d, d), 40, q_lo=q_lo, q_hi=q_hi, db_lo=db_lo, db_hi=db_hi)


@pytest.mark.parametrize("d", [20, 100])
def test_windows(engine, monkeypatch, d):
    monkeypatch.setenv("B200TSNE_KNN_WINDOW_TILES", "33")
    both(engine, monkeypatch, mixture(17000, d, 3), 33, q_lo=100, q_hi=1500)


@pytest.mark.parametrize("d", [20, 100])
def test_full_buffers(engine, monkeypatch, d):
    """3 000 copies of one point: more candidates than a buffer holds arrive from all blocks at once."""
    X = mixture(9000, d, 4)
    X[2000:5000] = X[2000]
    st = both(engine, monkeypatch, X, 50)
    assert st["rows_recomputed"] >= 3000


@pytest.mark.parametrize("pairs", ["bf16", "tf32"])
@pytest.mark.parametrize("d", [1, 4, 5, 9, 10, 15, 16, 20, 21, 25, 26, 31, 32, 36, 37, 42, 47, 48, 52, 53, 57, 58, 63])
def test_every_number_of_k_steps(engine, monkeypatch, d, pairs):
    """The narrow kernel's images: none to three groups of 16 dimensions and one to three steps for what is left."""
    monkeypatch.setenv("B200TSNE_KNN_FILTER", pairs)
    st = both(engine, monkeypatch, mixture(2300, d, 70 + d), 20)
    assert st["filter_error_ratio"] < 0.5 and st["rows_recomputed"] <= 46


@pytest.mark.parametrize("n,k", [(49151, 20), (49152, 20), (98303, 97), (98304, 97)])
def test_both_sides_of_rare_survivors(engine, monkeypatch, n, k):
    """From one key in 128 down the scan stores a lone survivor of eight behind a search for its place: every row, with
    points that repeat, so that survivors come alone, in pairs and in runs."""
    X = mixture(n, 5, k)
    X[: n // 7] = X[n // 2 : n // 2 + n // 7]
    st = both(engine, monkeypatch, X, k)
    assert st["rows_recomputed"] <= 0.02 * n
