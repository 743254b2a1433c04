"""Norms beyond the range of floats: every key of a sample is infinite, and the padding of the last tile must not pass."""
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
