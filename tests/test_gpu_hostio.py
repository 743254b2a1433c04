"""Host <-> device copies through the staging lanes: what goes in comes out, at the sizes where the path changes."""
import threading

import numpy as np
import pytest

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
