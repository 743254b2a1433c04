"""The exact search by whole rows of distances (csrc/knn_dense.cu): bit for bit the oracle's lists at the edges of its
tiles, of the keys a thread holds and of its segments, with exact ties, with fewer points than slots and for the rows the
tensor-core search hands over."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(n, d, seed, ties):
    rng = np.random.default_rng(seed)
    # small whole numbers: most distances occur many times and the order is decided by the index
    return rng.integers(0, 3, (n, d)).astype(np.float32) if ties else rng.normal(0, 1, (n, d)).astype(np.float32)


@pytest.mark.parametrize("ties", [False, True])
@pytest.mark.parametrize("n,d,k", [(1, 1, 1), (2, 3, 5), (63, 1, 64), (128, 33, 128), (129, 31, 20), (1024, 5, 90), (1025, 64, 91),
                                   (2047, 32, 512), (1500, 7, 513), (3000, 70, 40), (4097, 65, 33), (8193, 64, 16)])
def test_host_points(engine, oracle_cpu, n, d, k, ties):
    X = _points(n, d, n + d, ties)
    ids, d2 = engine.knn(X, k)
    lo = max(0, n - 700)                                     # the last rows: the ragged tiles
    ids_o, d2_o = oracle_cpu.knn(X, k, q_lo=lo, q_hi=n)
    if k > n:                                                # unfilled slots
        assert (ids[:, n:] == -1).all() and np.isinf(d2[:, n:]).all()
        ids, d2, ids_o, d2_o = ids[:, :n], d2[:, :n], ids_o[:, :n], d2_o[:, :n]
    assert np.array_equal(ids[lo:], ids_o) and np.array_equal(d2[lo:], d2_o)


@pytest.mark.parametrize("n,d,k,ties", [(300, 2, 4, False), (4099, 64, 16, False), (4099, 3, 60, True), (12288, 7, 32, True),
                                        (12289, 7, 32, True), (2000, 1000, 9, False)])
def test_device_points_without_allocation(engine, oracle_cpu, n, d, k, ties):
    import torch
    X = _points(n, d, n, ties)
    Xd = torch.from_numpy(X).cuda()
    ids = torch.empty(n, k, dtype=torch.int32, device="cuda")
    d2 = torch.empty(n, k, dtype=torch.float32, device="cuda")
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    engine.check(engine.lib.b200tsne_knn_noalloc(Xd.data_ptr(), n, d, k, ids.data_ptr(), d2.data_ptr(), C.c_void_p(st.cuda_stream)))
    st.synchronize()
    lo = n - min(n, 300)
    ids_o, d2_o = oracle_cpu.knn(X, k, q_lo=lo, q_hi=n)
    assert np.array_equal(ids.cpu().numpy()[lo:], ids_o) and np.array_equal(d2.cpu().numpy()[lo:], d2_o)


@pytest.mark.parametrize("n,k", [(12289, 16), (30011, 20), (70001, 40)])
def test_rows_handed_over_in_segments(engine, oracle_cpu, n, k):
    """Half of the points are copies of sixteen corners: neighbours beyond the last candidate are as near as the K-th, no
    such row can be certified, and each is searched in segments whose lists are merged."""
    X = np.random.default_rng(3).integers(0, 2, (n, 4)).astype(np.float32)
    X[: n // 2] += 0.25 * np.random.default_rng(1).random((n // 2, 4), dtype=np.float32)
    ids, d2 = engine.knn(X, k)
    st = engine.knn_last_stats()
    assert st["tensor_core"] == 1 and st["rows_recomputed"] > n // 4
    for lo in (0, n // 2 - 20, n - 60):
        ids_o, d2_o = oracle_cpu.knn(X, k, q_lo=lo, q_hi=lo + 60)
        assert np.array_equal(ids[lo:lo + 60], ids_o) and np.array_equal(d2[lo:lo + 60], d2_o)
