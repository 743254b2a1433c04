"""The exact search by whole rows of distances (csrc/knn_dense.cu): bit for bit the oracle's lists at the edges of its
tiles, of the keys a thread holds and of its segments, with exact ties, with fewer points than slots and for the rows the
tensor-core search hands over."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

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


@pytest.mark.parametrize("scale", [1e-19, 1e-20, 1e-21, 1e-22, 1e-23])
@pytest.mark.parametrize("n,d,k", [(300, 7, 20), (1500, 20, 32), (4099, 5, 50)])
def test_squares_at_the_end_of_the_range(engine, oracle_cpu, n, d, k, scale):
    """Squares that are subnormal or round to zero, where a fused operation could round otherwise than a product: blocks of 64
    queries, of 16 (at most 48 in all), and the search without allocation."""
    import torch
    X = (np.random.default_rng(n).normal(0, 1, (n, d)) * scale).astype(np.float32)
    ids_o, d2_o = oracle_cpu.knn(X, k, q_lo=n - 200, q_hi=n)
    for q_lo in (n - 200, n - 48, n - 1):
        ids, d2 = engine.knn(X, k, q_lo=q_lo, q_hi=n)
        assert np.array_equal(ids, ids_o[q_lo - n:]) and np.array_equal(d2, d2_o[q_lo - n:])
    ids, d2 = _noalloc(engine, torch.from_numpy(X).cuda(), k)
    assert np.array_equal(ids.cpu().numpy()[-200:], ids_o) and np.array_equal(d2.cpu().numpy()[-200:], d2_o)


# groups of four threads, of one, none (K = 48 / 49, 160 / 161); rows that bisect beyond K = 48 and longer ones; both sides of the
# numbers of keys a thread holds (test_selection_where_the_bound_is_loose has the others)
@pytest.mark.parametrize("k", [47, 48, 49, 160, 161, 192, 193])
@pytest.mark.parametrize("n", [256, 2047, 2048, 2049, 6144, 6145, 12288])
@pytest.mark.parametrize("equal", [0, 600])
def test_selection_by_a_bound(engine, oracle_cpu, n, k, equal):
    """Without ties, and with more equal distances below the bound than there is room for: decided by the index."""
    import torch
    X = _points(n, 3, n + k, False)
    X[n - min(n, equal):] = X[-1]
    Xd = torch.from_numpy(X).cuda()
    ids = torch.empty(n, k, dtype=torch.int32, device="cuda")
    d2 = torch.empty(n, k, dtype=torch.float32, device="cuda")
    engine.check(engine.lib.b200tsne_knn_noalloc(Xd.data_ptr(), n, 3, k, ids.data_ptr(), d2.data_ptr(), 0))
    torch.cuda.synchronize()
    lo = max(0, n - 300)
    ids_o, d2_o = oracle_cpu.knn(X, k, q_lo=lo, q_hi=n)
    assert np.array_equal(ids.cpu().numpy()[lo:], ids_o) and np.array_equal(d2.cpu().numpy()[lo:], d2_o)


def _awkward(n, d, kind):
    """Points for which the smallest keys of the selection's groups say little about the K-th smallest key."""
    rng = np.random.default_rng(n + d)
    if kind == "period":                                     # a class's points stand 256 rows apart
        return (rng.normal(0, 10, (256, d))[np.arange(n) % 256] + rng.normal(0, 1, (n, d))).astype(np.float32)
    if kind == "binary":
        return rng.integers(0, 2, (n, d)).astype(np.float32)
    X = rng.normal(0, 1, (n, d)).astype(np.float32)          # "copies": most points are one
    X[rng.random(n) < 0.8] = X[0]
    return X


def _noalloc(engine, Xd, k):
    import torch
    ids = torch.empty(len(Xd), k, dtype=torch.int32, device="cuda")
    d2 = torch.empty(len(Xd), k, dtype=torch.float32, device="cuda")
    engine.check(engine.lib.b200tsne_knn_noalloc(Xd.data_ptr(), *Xd.shape, k, ids.data_ptr(), d2.data_ptr(), torch.cuda.current_stream().cuda_stream))
    return ids, d2


# fewer keys than are ranked at once; a full block of places and one more; both sides of every number of keys a thread holds
@pytest.mark.parametrize("k", [16, 48, 90, 192, 300])
@pytest.mark.parametrize("n", [100, 256, 257, 1024, 1025, 4096, 4097, 6145, 8192, 8193, 12288])
@pytest.mark.parametrize("kind", ["period", "binary", "copies"])
def test_selection_where_the_bound_is_loose(engine, oracle_cpu, kind, n, k):
    import torch
    X, k = _awkward(n, 7, kind), min(k, n)
    ids, d2 = _noalloc(engine, torch.from_numpy(X).cuda(), k)
    lo = max(0, n - 100)
    ids_o, d2_o = oracle_cpu.knn(X, k, q_lo=lo, q_hi=n)
    assert np.array_equal(ids.cpu().numpy()[lo:], ids_o) and np.array_equal(d2.cpu().numpy()[lo:], d2_o)


@pytest.mark.parametrize("n,d,k", [(4099, 16, 90), (9000, 40, 16)])
@pytest.mark.parametrize("kind", ["period", "binary", "copies"])
def test_points_with_a_period_or_copies_take_no_longer(engine, kind, n, d, k):
    """Neither neighbours at equal steps in the array nor many equal distances cost more than a fifth (1.6 and 1.45 times as long
    where the bound is thrown away for them)."""
    import torch
    took = []
    for X in (np.random.default_rng(1).normal(0, 1, (n, d)).astype(np.float32), _awkward(n, d, kind)):
        Xd, times = torch.from_numpy(X).cuda(), []
        for _ in range(9):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(5):
                _noalloc(engine, Xd, k)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        took.append(sorted(times)[4])
    assert took[1] < 1.2 * took[0]


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


@pytest.mark.parametrize("n", [12288, 12289, 20011, 30000])
def test_rows_without_neighbours(n):
    """A row of NaN has no neighbours at any size: ids -1, distances +inf, in memory filled with other bits before (in a
    process of its own).  Nor does it change the others' affinities, which scale by 1 / 2N."""
    code = """
import numpy as np
from tsne_cuda_b200 import _lib as e
n, k = %d, 30
X = np.random.default_rng(n).normal(0, 1, (n, 20)).astype(np.float32)
X[-1] = np.nan
ids, d2 = e.knn(X, k)
assert (ids[-1] == -1).all() and np.isposinf(d2[-1]).all(), (ids[-1], d2[-1])
ids_r, d2_r = e.knn(X[:-1], k)
assert np.array_equal(ids[:-1], ids_r) and np.array_equal(d2[:-1], d2_r)
P = []
for x in (X, X[:-1]):
    with e.Session(len(x), k) as s:
        s.affinities_from_points(x, 10.0, 1e-4)
        P.append(s.get_affinities()[0][:n - 1].astype(np.float64) * len(x))
assert np.isfinite(P[0]).all() and np.abs(P[0] - P[1]).max() <= 2e-7 * P[1].max()
Y, Z = e.fit(X, num_neighbors=k, perplexity=10.0, iterations=20, random_seed=1)
assert np.isfinite(Y).all()
""" % n
    subprocess.run([sys.executable, "-c", code], check=True, cwd=ROOT, timeout=120, env=dict(os.environ, B200TSNE_POISON="1"))


def test_infinitely_far_neighbours_in_segments(engine):
    """Distances beyond the range of floats rank by id behind the finite ones, and before the slots that a segment of
    nothing but NaN leaves empty."""
    n, k, lo, hi = 25000, 24, 13000, 13040
    X = np.random.default_rng(2).normal(0, 1, (n, 8)).astype(np.float32) * np.float32(1e20)   # squared differences overflow
    X[:12500] = np.nan
    X[lo + 5] = X[lo + 4]
    ids, d2 = engine.knn(X, k, q_lo=lo, q_hi=hi)
    with np.errstate(over="ignore", invalid="ignore"):
        dist = np.zeros((hi - lo, n), np.float32)
        for d in range(8):
            t = X[lo:hi, None, d] - X[None, :, d]
            dist += t * t
    want = np.argsort(dist, axis=1, kind="stable")[:, :k]    # NaN last, equal distances by index
    assert np.array_equal(ids, want) and np.array_equal(d2, np.take_along_axis(dist, want, 1))
    assert (np.isfinite(d2).sum(1) < 4).all()


@pytest.mark.parametrize("n,k,copies", [(70001, 8, 2), (60000, 5, 2), (70001, 5, 24), (200003, 32, 2)])
def test_many_rows_handed_over_to_the_list_search(engine, oracle_cpu, n, k, copies):
    """Every `copies`-th point is one of sixteen corners: so many rows and pairs that lists are kept for them, over the whole
    database or in slices that are merged; a row of NaN among them stays empty."""
    X = np.random.default_rng(3).normal(0.5, 1, (n, 4)).astype(np.float32)
    X[::copies] = np.random.default_rng(4).integers(0, 2, (len(X[::copies]), 4))
    X[5 * copies] = np.nan
    ids, d2 = engine.knn(X, k)
    st = engine.knn_last_stats()
    assert st["tensor_core"] == 1 and st["rows_recomputed"] * n > 1e7 * k ** 1.5
    assert (ids[5 * copies] == -1).all() and np.isposinf(d2[5 * copies]).all()
    Xo = np.delete(X, 5 * copies, axis=0)                    # (the oracle takes no NaN)
    back = np.delete(np.arange(n), 5 * copies)
    for lo in (0, n // 2, n - 61):
        ids_o, d2_o = oracle_cpu.knn(Xo, k, q_lo=lo, q_hi=lo + 60)
        rows = back[lo:lo + 60]
        assert np.array_equal(ids[rows], back[ids_o]) and np.array_equal(d2[rows], d2_o)


@pytest.mark.parametrize("ties", [False, True])
@pytest.mark.parametrize("n,d,k", [(300, 20, 10), (2047, 50, 90), (9000, 20, 300), (12289, 7, 256), (32768, 5, 230)])
def test_against_the_list_search_on_every_row(engine, monkeypatch, n, d, k, ties):
    """Whole rows of distances against the search that keeps lists (forced at any size), which shares no kernel with it."""
    X = _points(n, d, n + k, ties)
    ids, d2 = engine.knn(X, k)
    assert engine.knn_last_stats()["tensor_core"] == 0
    monkeypatch.setenv("B200TSNE_KNN", "simt")
    ids_l, d2_l = engine.knn(X, k)
    assert np.array_equal(ids, ids_l) and np.array_equal(d2, d2_l)


@pytest.mark.parametrize("n,rows", [(2147, 2147), (2305, 2305), (2305, 48), (2305, 49), (20000, 48), (32768, 37)])
@pytest.mark.parametrize("d", [1, 32, 33, 97])
def test_distances_on_both_sides_of_four_blocks_to_an_sm(engine, monkeypatch, n, rows, d):
    """592 blocks of 64 (16 from 48 rows on down) queries and 128 points on 148 SMs: 578, 703, 57, 19, 471 and 768 here."""
    X = _points(n, d, n + d, False)
    lo = (n - rows) // 2
    ids, d2 = engine.knn(X, 240, lo, lo + rows)
    assert engine.knn_last_stats()["tensor_core"] == 0
    monkeypatch.setenv("B200TSNE_KNN", "simt")
    ids_l, d2_l = engine.knn(X, 240, lo, lo + rows)
    assert np.array_equal(ids, ids_l) and np.array_equal(d2, d2_l)


@pytest.mark.parametrize("n,d,k", [(700, 33, 20), (4099, 64, 16), (9000, 20, 150)])
def test_a_search_between_the_kernels_that_write_and_clear_its_points(engine, n, d, k):
    """The rounds of a search overlap with each other, but not with what the caller has queued before and after it in the
    stream: queued, and captured with its producer."""
    import torch
    stream = torch.cuda.Stream()
    source, X = torch.empty(n, d, device="cuda"), torch.empty(n, d, device="cuda")
    ids, d2 = torch.empty(n, k, dtype=torch.int32, device="cuda"), torch.empty(n, k, device="cuda")

    def search():
        engine.check(engine.lib.b200tsne_knn_noalloc(X.data_ptr(), n, d, k, ids.data_ptr(), d2.data_ptr(), stream.cuda_stream))

    def expect(points):
        want_i, want_d = _noalloc(engine, points, k)
        assert torch.equal(ids, want_i) and torch.equal(d2, want_d)

    for _ in range(3):
        with torch.cuda.stream(stream):
            source.normal_()
            slow = torch.ones(3000, 3000, device="cuda") @ torch.ones(3000, 3000, device="cuda")   # the points come late
            torch.mul(source, slow[0, 0] / 3000, out=X)
            search()
            points = X.clone()
            X.zero_()
        torch.cuda.synchronize()
        expect(points)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        torch.mul(source, 2.0, out=X)
        search()
        X.zero_()
    for _ in range(3):
        source.normal_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        expect(2.0 * source)
