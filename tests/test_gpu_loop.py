"""The gradient loop at the sizes where its kernels change, and the early stop taken on the device.

Bars: one iteration against the CPU oracle.  The update is  u = m u0 - eta g (a F_attr - F_rep / Z); the forces are within
1e-5 and 1e-4 of the oracle (relative L2, test_gpu_stages.py), so the new momentum from u0 = 0 is within their sum."""
import time

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _graph(n, k, seed):
    rng = np.random.default_rng(seed)
    ids = rng.integers(0, n, (n, k), dtype=np.int32)
    P = (rng.random((n, k)) / (n * k)).astype(np.float32)
    return P, ids, rng


def _same(a, b):
    """Embedding and momentum up to the order of the forces' sums.  A gain takes its other value (a fifth away) where that
    turns the sign of a gradient near zero: at most one coordinate in 10^4."""
    assert rel_l2(a[0], b[0]) < 1e-6 and rel_l2(a[1], b[1]) < 1e-6
    assert (np.abs(a[2] - b[2]) > 1e-5).mean() < 1e-4 and a[3] == b[3]


# the first iteration: points one by one up to 2,999, a point a lane in the order as it is allocated up to 131,072, sorted from
# 65,536 on; then four a lane
@pytest.mark.parametrize("n", [1, 31, 8192, 8193, 32767, 32768, 131072, 131075])
@pytest.mark.parametrize("spread", [1e-4, 20.0])
def test_one_iteration_vs_oracle(engine, oracle_cpu, n, spread):
    P, ids, rng = _graph(n, 4, n)
    Y = rng.normal(0, spread, (2, n)).astype(np.float32)
    Y[:, : n // 3] *= 0.02                                   # a dense part: long runs of points in one box
    with engine.Session(n, 4) as s:
        s.set_affinities(P, ids)
        s.set_schedule(100.0, 12.0, 250, 0.5, 0.8)
        s.set_embedding(Y)
        s.run(1)
        Y1, mom, gains, step = s.get_state()
    Yo, gains_o, mom_o, _ = oracle_cpu.iterate(P, ids, Y, 1, 100.0)
    assert step == 1
    if n == 1:                                               # no neighbour but itself, Z = 0: nothing finite to compare
        return
    assert rel_l2(mom, mom_o) < 1.1e-4
    # the embedding rounds once more per coordinate
    assert np.abs(Y1 - Yo).max() < 1.1e-4 * np.linalg.norm(mom_o) + 2e-7 * np.abs(Yo).max()


# Exaggerated: one by one below 3,000 points, then through an order that is sorted beside the chain every eighth iteration, from
# 32,768 on every fourth, from 65,536 on on the chain in each.  Settled: one by one up to 8,192, merged in natural order below
# 32,768, then sorted beside the chain.  Both sides of every border, after single steps, pairs and blocks.
@pytest.mark.parametrize("n", [2999, 3000, 8192, 8193, 32767, 32768, 65535, 65536, 131072, 131075])
@pytest.mark.parametrize("step", [0, 400])
@pytest.mark.parametrize("before", [[1], [1] * 9, [2] * 9, [64, 2]])
def test_an_iteration_through_a_refreshed_order_vs_oracle(engine, oracle_cpu, n, step, before):
    """One more iteration from wherever some have led, so that it spreads the points in the order that those have sorted."""
    P, ids, rng = _graph(n, 4, n)
    Y = rng.normal(0, 1e-4 if step == 0 else 20.0, (2, n)).astype(np.float32)
    Y[:, : n // 3] *= 0.02
    with engine.Session(n, 4) as s:
        s.set_affinities(P, ids)
        s.set_schedule(100.0, 12.0, 250, 0.5, 0.8)
        s.set_state(Y, np.zeros_like(Y), np.ones_like(Y), step)
        for k in before:
            s.run(k)
        Y0, u0, g0, at = s.get_state()
        s.run(1)
        Y1, u1, g1, _ = s.get_state()
    assert at == step + sum(before)
    _, g_o, u_o, _ = oracle_cpu.iterate(P, ids, Y0, 1, 100.0, first_step=at, gains=g0, old=u0)
    m = np.float32(0.5 if at < 250 else 0.8)
    # the new part of the momentum is the forces', the rest rounds once
    assert np.linalg.norm((u1 - m * u0) - (u_o - m * u0)) < 1.1e-4 * np.linalg.norm(u_o - m * u0) + 2.0 ** -23 * np.linalg.norm(u0)
    assert (np.abs(g1 - g_o) > 1e-5).mean() < 1e-3 and np.abs(Y1 - (Y0 + u1)).max() <= 2.0 ** -23 * np.abs(Y1).max()


@pytest.mark.parametrize("n", [3000, 8193, 32768, 65535])
@pytest.mark.parametrize("step", [0, 400])
def test_order_beside_the_chain_and_none_agree(engine, monkeypatch, n, step):
    """40 iterations from a blob (settled: from a layout) through orders sorted beside the chain, sorted on it in each iteration,
    and in natural order: up to the order of the sums, as between blocks and single steps below."""
    P, ids, rng = _graph(n, 6, 6)
    Y = rng.normal(0, 1e-4 if step == 0 else 5.0, (2, n)).astype(np.float32)
    out = []
    for refresh, early in ((None, None), ("1", "1"), ("0", None)):
        for name, value in (("B200TSNE_ORDER_REFRESH", refresh), ("B200TSNE_ORDER_REFRESH_EARLY", early)):
            if value is None:
                monkeypatch.delenv(name, raising=False)
            else:
                monkeypatch.setenv(name, value)
        with engine.Session(n, 6) as s:
            s.set_affinities(P, ids)
            s.set_schedule(1.0, 12.0, 250, 0.5, 0.8)
            s.set_state(Y, np.zeros_like(Y), np.ones_like(Y), step)
            s.run(40)
            out.append(s.get_state())
    for o in out[1:]:
        assert rel_l2(o[0], out[0][0]) < 1e-6 and rel_l2(o[1], out[0][1]) < 1e-4


@pytest.mark.parametrize("n", [700, 40000])
@pytest.mark.parametrize("stop_after", [1, 2, 5, 16, 17, 20])
def test_stop_on_the_device_takes_place_where_the_host_would(engine, n, stop_after):
    """Momentum that fades makes the update norm fall from step to step: the run ends after the first iteration whose
    norm is below the threshold, whatever block it was queued in, and the loop goes on from there."""
    P, ids, rng = _graph(n, 6, 5)
    Y = rng.normal(0, 5.0, (2, n)).astype(np.float32)
    mom = rng.normal(0, 1.0, (2, n)).astype(np.float32)

    def session():
        s = engine.Session(n, 6)
        s.set_affinities(P, ids)
        s.set_schedule(1e-3, 12.0, 250, 0.8, 0.8)
        s.set_state(Y, mom, np.ones_like(mom), 0)
        return s

    with session() as s:
        norms = []
        for _ in range(24):
            s.run(1, min_gradient_norm=1e-30)
            norms.append(s.stats()["update_norm"])
    assert all(a > b for a, b in zip(norms, norms[1:]))
    threshold = 0.5 * (norms[stop_after - 1] + (norms[stop_after - 2] if stop_after > 1 else 2 * norms[0]))
    with session() as s, session() as t:
        _, done = s.run(23, min_gradient_norm=threshold)
        assert done == stop_after and s.stats()["step"] == stop_after
        assert abs(s.stats()["update_norm"] / norms[stop_after - 1] - 1) < 1e-5
        t.run(stop_after)
        _same(s.get_state(), t.get_state())
        assert abs(s.stats()["Z"] / t.stats()["Z"] - 1) < 1e-5
        s.run(7)
        t.run(7)
        _same(s.get_state(), t.get_state())


def test_blocks_of_iterations_and_single_steps_agree(engine):
    """Captured blocks of 16, pairs and single steps, across the phases of the schedule, against direct launches."""
    n = 40000                                                # sorted: the late phase sorts every eighth iteration
    P, ids, rng = _graph(n, 6, 6)
    Y = rng.normal(0, 5.0, (2, n)).astype(np.float32)
    out = []
    for chunks in ([57], [1] * 57, [16, 3, 2, 1, 35], [57]):
        with engine.Session(n, 6) as s:
            s.set_affinities(P, ids)
            s.set_schedule(1.0, 12.0, 18, 0.5, 0.8)
            s.set_state(Y, np.zeros_like(Y), np.ones_like(Y), 3)
            if len(out) == 3:
                s.enable_stage_timers(True)                  # direct launches, the gather a kernel of its own
            for c in chunks:
                s.run(c)
            out.append(s.get_state())
    for o in out[1:]:
        assert o[3] == out[0][3] == 60
        assert rel_l2(o[0], out[0][0]) < 1e-6 and rel_l2(o[1], out[0][1]) < 1e-4


@pytest.mark.parametrize("n,step,refresh,early,chunks,sorts", [
    (40000, 400, "32", None, [64, 64], 4),                   # a period above a block's sixteen iterations
    (40000, 400, "10", None, [160], 16),                     # one that does not divide them
    (40000, 400, "10", None, [1] * 40, 4),
    (40000, 400, "5", None, [2] * 20, 8),
    (40000, 400, None, None, [64], 8),
    (40000, 0, "0", "1", [64], 0),                           # natural order, whatever the other variable says
    (20000, 0, None, "4", [64], 16),
    (2999, 0, None, None, [64], 0),
    (3000, 0, None, None, [64], 8),
    (65535, 0, None, None, [64], 16),
    (65536, 0, None, None, [64], 64),
])
def test_how_often_the_order_is_sorted(engine, monkeypatch, n, step, refresh, early, chunks, sorts):
    """Counted in launches: a sort has three."""
    P, ids, rng = _graph(n, 3, 4)
    Y = rng.normal(0, 5.0, (2, n)).astype(np.float32)

    def launches():
        with engine.Session(n, 3) as s:
            s.set_affinities(P, ids)
            s.set_schedule(1e-3, 12.0, 250, 0.5, 0.8)
            s.set_state(Y, np.zeros_like(Y), np.ones_like(Y), step)
            before = s.launch_count()
            for c in chunks:
                s.run(c)
            return s.launch_count() - before

    for name, value in (("B200TSNE_ORDER_REFRESH", refresh), ("B200TSNE_ORDER_REFRESH_EARLY", early)):
        if value is None:
            monkeypatch.delenv(name, raising=False)
        else:
            monkeypatch.setenv(name, value)
    got = launches()
    monkeypatch.setenv("B200TSNE_ORDER_REFRESH", "0")
    monkeypatch.delenv("B200TSNE_ORDER_REFRESH_EARLY", raising=False)
    assert got - launches() == 3 * sorts


def _steps(engine, monkeypatch, n, graphs, per_call, decay):
    monkeypatch.setenv("B200TSNE_GRAPHS", "1" if graphs else "0")
    P, ids, rng = _graph(n, 6, 8)
    Y = rng.normal(0, 5.0, (2, n)).astype(np.float32)
    with engine.Session(n, 6) as s:
        s.set_affinities(P, ids)
        s.set_state(Y, np.zeros_like(Y), np.ones_like(Y), 0)
        t = []
        for k in range(60):
            s.set_schedule(1.0 * (0.98 ** k if decay else 1.0), 12.0, 250, 0.5, 0.8)
            t0 = time.perf_counter()
            s.run(per_call)
            t.append(time.perf_counter() - t0)
        return sorted(t)[30], s.get_state()


@pytest.mark.parametrize("n", [2000, 60000])
@pytest.mark.parametrize("per_call", [1, 2, 3])
def test_a_schedule_that_changes_at_every_call_is_not_captured_every_time(engine, monkeypatch, n, per_call):
    """A block is captured when it serves again: calls that each bring another learning rate take the time of direct
    launches (a capture and an executable in each call: 2.4 to 3.7 times that; the bar leaves half for a busy host), and
    calls that repeat a schedule end up below it (0.6 to 0.9 of it; a tenth for the host)."""
    direct, a = _steps(engine, monkeypatch, n, False, per_call, True)
    changing, b = _steps(engine, monkeypatch, n, True, per_call, True)
    repeated, _ = _steps(engine, monkeypatch, n, True, per_call, False)
    # the bars of the test above: an iteration's forces round to 1e-7 in no fixed order and the loop carries it on, so
    # after up to 180 of them (57 there) momentum is held to 1e-4, which another eta in one call (2 %) exceeds by far
    assert rel_l2(a[0], b[0]) < 1e-6 and rel_l2(a[1], b[1]) < 1e-4 and a[3] == b[3]
    assert changing < 1.5 * direct and repeated < 1.1 * direct


def test_a_session_after_many_kinds_of_others_finds_its_executables(engine):
    """Sessions of several sizes, phases and steps leave more executables than the sixteen that are kept.  The first session of
    another size pays for its own (3 ms on 5.6), the second finds them (its first run 1.03 of the others; made anew, 1.5)."""
    def session(n):
        P, ids, rng = _graph(n, 6, n)
        Y = rng.normal(0, 5.0, (2, n)).astype(np.float32)
        s = engine.Session(n, 6)
        s.set_affinities(P, ids)
        s.set_schedule(1.0, 12.0, 250, 0.5, 0.8)
        return s, lambda step: s.set_state(Y, np.zeros_like(Y), np.ones_like(Y), step)

    engine.release_cached_memory()                            # one set of streams, nothing kept
    for n in (2000, 4000, 70000, 140000):
        s, start = session(n)
        with s:
            for step in (0, 400):
                start(step)
                for per in [64, 64] + [1] * 20 + [2] * 20:
                    s.run(per)
    for _ in range(2):
        s, start = session(40000)
        with s:
            t = []
            for _ in range(7):
                start(0)
                t0 = time.perf_counter()
                s.run(224)
                t.append(time.perf_counter() - t0)
    assert t[0] < 1.15 * sorted(t)[3]


@pytest.mark.parametrize("n", [1, 33, 21845, 21846])
def test_state_goes_in_and_out_unchanged(engine, n):
    """Both sides of the largest state that crosses in one piece; a second state right behind the first."""
    P, ids, rng = _graph(n, 3, n)
    a, b = [[rng.normal(0, 1, (2, n)).astype(np.float32) for _ in range(3)] for _ in range(2)]
    with engine.Session(n, 3) as s:
        s.set_affinities(P, ids)
        s.set_state(*a, 4)
        s.set_state(*b, 7)
        got = s.get_state()
        assert got[3] == 7 and all(np.array_equal(x, y) for x, y in zip(got, b))
        assert np.array_equal(s.get_embedding(), b[0])
        s.set_state(*a, 9)
        s.run(1)
        Y, u, _, step = s.get_state()
        assert step == 10 and np.array_equal(Y, a[0] + u)    # the step was taken from the first state


@pytest.mark.parametrize("n", [2000, 21846])
@pytest.mark.parametrize("where", ["YMG", "Y", "G"])
def test_state_in_device_memory(engine, n, where):
    """Arrays of a state may stand in device memory, some or all of them, at any size."""
    import ctypes as C

    import torch
    P, ids, rng = _graph(n, 3, n)
    host = [rng.normal(0, 1, (2, n)).astype(np.float32) for _ in range(3)]

    def at(arrays):
        return [C.cast(a.data_ptr() if torch.is_tensor(a) else a.ctypes.data, C.POINTER(C.c_float)) for a in arrays]

    def there(arrays):
        return [torch.from_numpy(a).cuda() if k in where else a.copy() for k, a in zip("YMG", arrays)]

    with engine.Session(n, 3) as s:
        s.set_affinities(P, ids)
        given = there(host)
        torch.cuda.synchronize()
        engine.check(engine.lib.b200tsne_session_set_state(s._h, *at(given), 4))
        got = s.get_state()
        assert got[3] == 4 and all(np.array_equal(a, b) for a, b in zip(got, host))
        out = there([np.zeros_like(a) for a in host])
        torch.cuda.synchronize()
        step = C.c_int()
        engine.check(engine.lib.b200tsne_session_get_state(s._h, *at(out), C.byref(step)))
        torch.cuda.synchronize()
        assert step.value == 4 and all(np.array_equal(torch.as_tensor(a).cpu().numpy(), b) for a, b in zip(out, host))
        Y = there([np.zeros_like(host[0])])[0]
        torch.cuda.synchronize()
        engine.check(engine.lib.b200tsne_session_get_embedding(s._h, at([Y])[0]))
        torch.cuda.synchronize()
        assert np.array_equal(torch.as_tensor(Y).cpu().numpy(), host[0])


@pytest.mark.parametrize("n", [2000, 21845, 21846])
def test_set_state_returns_when_the_state_has_arrived(engine, n):
    """Nothing is left on the device when set_state returns: waiting for it takes what waiting for an idle device does (half
    a megabyte still on its way: 30 us more)."""
    import torch
    P, ids, rng = _graph(n, 3, n)
    a = [rng.normal(0, 1, (2, n)).astype(np.float32) for _ in range(3)]
    left, idle = [], []
    with engine.Session(n, 3) as s:
        s.set_affinities(P, ids)
        for _ in range(301):
            s.set_state(*a, 4)
            for t in (left, idle):
                t0 = time.perf_counter()
                torch.cuda.synchronize()
                t.append(time.perf_counter() - t0)
    assert sorted(left)[150] < 1.5 * sorted(idle)[150] + 2e-6
