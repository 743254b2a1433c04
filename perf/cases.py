"""Timed cases of the engine: what a user's program has it do, through the entry points it would call.

Four kinds of work:

  fit         host points in, host embedding out: TSNE.fit_transform (or _lib.fit where the start is drawn from a seed).
              Neighbour search, affinities and the gradient loop in one call: what nearly every user runs.
  session     _lib.Session, the device-resident loop: a checkpoint goes in, some iterations run, the state comes back.
              Resuming, stepping an interactive view, iterating on a neighbour graph that was computed elsewhere.
  knn         _lib.knn: the exact neighbour lists of host points, for programs that only want the graph.
  knn_device  b200tsne_knn_noalloc: the same for a few points in device memory, queued on the caller's stream.

Points are drawn on the GPU in three shapes: Gaussian clusters, images (most pixels exactly zero) and rectified
classifier features.  Embeddings that a call starts from are layouts such as an earlier run leaves behind: one disc per
class, points placed in it by a projection of their coordinates.
"""
import math

import numpy as np
import torch

from tsne_cuda_b200 import TSNE, _lib

GRID_NODES = 390 * 390


def _fit(name, n, d, data, classes, k, perplexity, iters, exag_iters, lr=200.0, start="layout", returns="once", min_grad=0.0):
    return dict(name=name, kind="fit", n=n, d=d, data=data, classes=classes, k=k, perplexity=perplexity, iters=iters,
                exag_iters=exag_iters, lr=lr, start=start, returns=returns, min_grad=min_grad)


def _session(name, n, d, data, classes, k, perplexity, iters, step, lr=200.0, graph="points"):
    return dict(name=name, kind="session", n=n, d=d, data=data, classes=classes, k=k, perplexity=perplexity, iters=iters,
                step=step, lr=lr, graph=graph)


def _knn(name, kind, n, d, data, classes, k):
    return dict(name=name, kind=kind, n=n, d=d, data=data, classes=classes, k=k)


def listed():
    return [
        # an interactive view of a small map asks for one more iteration and draws it: latency and launches only
        _session("view_2k", 2000, 50, "mixture", 4, 90, 30.0, iters=1, step=500),
        # a few rows of a table: the shortest whole fit
        _fit("fit_1500", 1500, 20, "mixture", 6, 32, 10.0, iters=250, exag_iters=250, lr=10.0),
        # a small map resumed from a checkpoint in its second phase and run on
        _session("resume_5k", 5000, 50, "mixture", 4, 90, 30.0, iters=200, step=500, lr=10.0),
        # an odd number of images, frames of the run kept for an animation, stopped by the gradient norm if it gets there
        _fit("fit_20k_snapshots", 20011, 784, "pixels", 10, 90, 30.0, iters=200, exag_iters=150, lr=10.0, returns="snapshots",
             min_grad=1e-7),
        # a graph computed elsewhere (ragged size, no points to order it by), embedded from a layout
        _session("graph_30k", 30011, 32, "mixture", 10, 64, 20.0, iters=100, step=0, lr=100.0, graph="given"),
        # an image collection of the usual size in the exaggerated phase
        _session("resume_60k", 60000, 784, "pixels", 10, 90, 30.0, iters=100, step=100),
        # the same collection from its pixels to the map
        _fit("fit_60k_images", 60000, 784, "pixels", 10, 90, 30.0, iters=250, exag_iters=250),
        # classifier features, embedded from a seeded random start: the widest points, the longest neighbour lists
        _fit("fit_50k_features", 50000, 1024, "features", 10, 150, 50.0, iters=250, exag_iters=250, lr=10.0, start="seed"),
        # a million points: the benchmark's size, whole and then the loop alone in its second phase
        _fit("fit_1m", 1000000, 50, "mixture", 4, 90, 30.0, iters=250, exag_iters=250),
        _session("resume_1m", 1000000, 50, "mixture", 4, 90, 30.0, iters=100, step=500, lr=1000.0),
        # the graph alone, an odd number of embedding vectors
        _knn("knn_100k", "knn", 100003, 96, "mixture", 30, 32),
        # a service's small batch of vectors, already on the device
        _knn("knn_4k_device", "knn_device", 4099, 64, "mixture", 10, 16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# the pair-dimensions of one exact search: the largest listed case has 5e13 of them, in clustered points where much of
# the data can be skipped; drawn ones stay below that, points of any shape scanned in full well below
_SEARCH_NARROW, _SEARCH_WIDE = 2.0e13, 5.0e12


def _points_shape(rng, n_lo, n_hi):
    """n, d, data, classes within what the largest listed search costs."""
    data = rng.choice(["mixture", "mixture", "pixels", "features"])
    n = _log_int(rng, n_lo, n_hi)
    d_hi = min(1024.0, 4.0e7 / n, (_SEARCH_NARROW if n > 200000 else _SEARCH_WIDE) / (float(n) * n))
    if n > 200000:
        d_hi = min(d_hi, 63.0)
    if data != "mixture" and d_hi < 64:
        data = "mixture"      # a handful of pixels or activations is nothing but repeated points
    d = _log_int(rng, 8 if data == "mixture" else 64, max(9.0, d_hi))
    return n, d, data, rng.choice([2, 4, 10, 30])


def draw(rng):
    kind = rng.choice(["fit", "fit", "session", "session", "knn", "knn_device"])
    if kind == "knn_device":
        d = _log_int(rng, 2, 128)
        return dict(kind=kind, n=_log_int(rng, 300, min(10000, (4 << 20) // d)), d=d, data="mixture", classes=rng.choice([2, 10]),
                    k=rng.randint(4, 64))
    if kind == "knn":
        n, d, data, classes = _points_shape(rng, 1000, 300000)
        return dict(kind=kind, n=n, d=d, data=data, classes=classes, k=rng.randint(5, 150))
    perplexity = float(rng.randint(5, 50))
    k = 3 * int(perplexity) if perplexity > 12 else rng.choice([32, 3 * int(perplexity)])
    n, d, data, classes = _points_shape(rng, 1000, 600000)
    case = dict(kind=kind, n=n, d=d, data=data, classes=classes, k=k, perplexity=perplexity, lr=float(min(200, max(10, n // 2000))))
    if kind == "session":
        case.update(iters=_log_int(rng, 1, 200 if n < 200000 else 100), step=rng.choice([0, 100, 300, 500, 777]),
                    graph=rng.choice(["points", "points", "given"]))
    else:
        iters = rng.randint(50, 250)
        case.update(iters=iters, exag_iters=rng.choice([250, iters - 40]), returns=rng.choice(["once", "once", "snapshots"]),
                    start="seed" if n > 200000 and rng.random() < 0.5 else "layout", min_grad=rng.choice([0.0, 0.0, 1e-7]))
        if case["start"] == "seed":
            case.update(returns="once", exag_iters=250)
    return case


# ---- inputs --------------------------------------------------------------------------------------
def _points(case, g):
    """(X (n, d) on the GPU, class of every row, what sets a row apart from its class (n, d))."""
    n, d, classes = case["n"], case["d"], case["classes"]
    rows = torch.randperm(n, generator=g, device="cuda") % classes
    if case["data"] == "pixels":      # values in [0, 1], four in five pixels of a class always zero
        mask = torch.rand(classes, d, generator=g, device="cuda") >= 0.8
        mask[:, 0] = True
        proto = torch.rand(classes, d, generator=g, device="cuda") * mask
        rest = 0.1 * torch.randn(n, d, generator=g, device="cuda")
        rest *= mask[rows]
        X = (proto[rows] + rest).clamp_(0.0, 1.0)
    elif case["data"] == "features":  # rectified class activations
        mu = torch.randn(classes, d, generator=g, device="cuda")
        rest = torch.randn(n, d, generator=g, device="cuda")
        X = (mu[rows] + rest).clamp_(min=0.0)
    else:                             # unit clusters, centres ten units apart in each coordinate
        mu = 10.0 * torch.randn(classes, d, generator=g, device="cuda")
        rest = torch.randn(n, d, generator=g, device="cuda")
        X = mu[rows] + rest
    return X.contiguous(), rows, rest


def _layout(case, rows, rest, g):
    """(2, n): the classes as discs on a ring, a point's place in its disc from two projections of `rest`."""
    classes = case["classes"]
    axes = torch.randn(rest.shape[1], 2, generator=g, device="cuda")
    t = (rest.double() @ axes.double()).float()
    t = t / t.std(dim=0, keepdim=True).clamp_min(1e-20)
    r2 = (t * t).sum(dim=1, keepdim=True)
    t = t * torch.sqrt((1.0 - torch.exp(-0.5 * r2)) / r2.clamp_min(1e-12))     # Gaussian -> even in the unit disc
    angle = 2.0 * math.pi * torch.arange(classes, device="cuda") / classes
    ring = torch.stack([torch.cos(angle), torch.sin(angle)], dim=1) * 12.0
    radius = 12.0 * min(0.9, 0.9 * math.sin(math.pi / classes)) if classes > 1 else 12.0
    return (ring[rows] + radius * t).t().contiguous()


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 2654435761 % (1 << 62))
    X, rows, rest = _points(case, g)
    st = {"case": case}
    if case["kind"] == "knn_device":
        st["X"] = X
        st["ids"] = torch.empty(case["n"], case["k"], dtype=torch.int32, device="cuda")
        st["d2"] = torch.empty(case["n"], case["k"], dtype=torch.float32, device="cuda")
        return st
    st["X"] = X.cpu().numpy()
    if case["kind"] == "knn":
        return st
    Y = _layout(case, rows, rest, g).cpu().numpy()
    del X, rows, rest
    if case["kind"] == "fit":
        st["y"] = np.asfortranarray(Y.T)
        st["seed"] = 1 + int(seed) % 1000000
        st["tsne"] = TSNE(perplexity=case["perplexity"], num_neighbors=case["k"], learning_rate=case["lr"], n_iter=case["iters"],
                          force_magnify_iters=case["exag_iters"], return_style=case["returns"], min_grad_norm=case["min_grad"])
        return st
    s = _lib.Session(case["n"], case["k"])
    if case["graph"] == "given":
        with _lib.Session(case["n"], case["k"]) as other:
            other.affinities_from_points(st["X"], case["perplexity"], 1e-3)
            st["P"], st["neighbours"] = other.get_affinities()
    else:
        s.affinities_from_points(st["X"], case["perplexity"], 1e-3)
    s.set_schedule(case["lr"], 12.0, 250, 0.5, 0.8)
    st.update(session=s, Y=Y, momentum=np.zeros_like(Y), gains=np.ones_like(Y))
    del st["X"]
    return st


# ---- one pass ------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    if case["kind"] == "fit":
        if case["start"] == "seed":
            return _lib.fit(state["X"], random_seed=state["seed"], perplexity=case["perplexity"], num_neighbors=case["k"],
                            learning_rate=case["lr"], iterations=case["iters"], force_magnify_iters=case["exag_iters"],
                            min_gradient_norm=case["min_grad"])[0]
        return state["tsne"].fit_transform(state["X"], state["y"])
    if case["kind"] == "session":
        s = state["session"]
        if case["graph"] == "given":
            s.set_affinities(state["P"], state["neighbours"])
        s.set_state(state["Y"], state["momentum"], state["gains"], case["step"])
        s.run(case["iters"])
        if case["iters"] > 30:
            return s.get_embedding()
        Y, momentum, gains, _ = s.get_state()
        return {"embedding": Y, "momentum": momentum, "gains": gains}
    if case["kind"] == "knn":
        ids, d2 = _lib.knn(state["X"], case["k"])
        return {"ids": ids, "d2": d2}
    X = state["X"]
    _lib.check(_lib.lib.b200tsne_knn_noalloc(X.data_ptr(), case["n"], case["d"], case["k"], state["ids"].data_ptr(),
                                             state["d2"].data_ptr(), torch.cuda.current_stream().cuda_stream))
    return {"ids": state["ids"], "d2": state["d2"]}


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    n, d, k = float(case["n"]), float(case["d"]), float(case["k"])
    search = {"bytes": 4.0 * n * d + 8.0 * n * k, "flops": 2.0 * n * n * d}
    if case["kind"] in ("knn", "knn_device"):
        return search
    # an iteration: value and id of every stored neighbour, the points' state, three passes over the four-term grid
    loop = case["iters"] * (8.0 * n * k + 104.0 * n + 48.0 * GRID_NODES)
    flops = case["iters"] * n * (12.0 * k + 150.0)
    if case["kind"] == "session":
        given = 8.0 * n * k if case["graph"] == "given" else 0.0
        return {"bytes": loop + 48.0 * n + given, "flops": flops}
    return {"bytes": search["bytes"] + loop + 16.0 * n, "flops": search["flops"] + flops}


def tolerance(case):
    if case["kind"] in ("knn", "knn_device"):
        return "exact"        # the distances are defined operation by operation, the order by (distance, id)
    # An iteration rounds its forces to about 1e-7 and sums them in no fixed order, and the loop multiplies that: a
    # coordinate's gain takes another value when the sign of a gradient near zero turns.  Repeated runs of these cases
    # differ by up to 3e-4 in the embedding after all iterations, at single points by a hundredth of its size.
    if case["kind"] == "session" and case["iters"] <= 30:
        return {"rel": 2e-3, "max": 0.9}      # gains are among the outputs: steps of a fifth at single coordinates
    return {"rel": 5e-4, "max": 0.05}
