"""The calls a program built on this framework makes, as cases that can be timed.

A case is one pass through the public entry points of ``hrnn_b200``: building an
index (HNSW insertion, NNDescent refinement, reverse lists), growing it with
dynamic inserts, answering RkNN queries one at a time, in batches and through
captured plans, in each precision, the learned budget's gradients, and the
transpose of a caller-owned KNN graph.  Data are seeded Gaussian mixtures (centres
N(0, 4 I), sigma 1), the distribution the benchmark and the tests use.

A serving program builds its index once and answers many batches from it: the
search cases keep one index per set of index sizes, and a seed makes other
queries, not another index.  The build cases make the points themselves from the
seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import hrnn_b200 as H

M, EFC, SAMPLE, NEAR = 16, 400, 50, 10  # links, construction beam, NNDescent sample, k of RkNN


def listed():
    return [
        # one interactive query on a small index, host call: launches and latency
        {"name": "one-query", "kind": "search", "form": "exact", "call": "host", "n": 20000, "d": 128, "K": 100,
         "nq": 1, "m": 5, "m_to": 5, "ef": 200, "ef_to": 200},
        # a web request's worth of queries at an ordinary embedding width that is no
        # multiple of 16, host arrays, the exact form
        {"name": "batch-d100", "kind": "search", "form": "exact", "call": "host", "n": 20011, "d": 100, "K": 60,
         "nq": 333, "m": 5, "m_to": 5, "ef": 128, "ef_to": 128},
        # an offline job: a large batch in the exact form, everything on the device
        {"name": "exact-10k", "kind": "search", "form": "exact", "call": "device", "n": 300000, "d": 128, "K": 500,
         "nq": 10000, "m": 5, "m_to": 5, "ef": 200, "ef_to": 200},
        # queries that each bring their own m and ef, BF16 form, wide rows
        {"name": "uneven-bf16-d256", "kind": "search", "form": "bf16", "call": "device", "n": 100000, "d": 256,
         "K": 200, "nq": 3000, "m": 1, "m_to": 50, "ef": 50, "ef_to": 400},
        # the serving loop at full size: the benchmark's 1M x 128, K_knng = 500 index,
        # 10,000 queries per replay of a captured plan, INT8 form
        {"name": "plan-int8-1M", "kind": "search", "form": "int8", "call": "plan", "n": 1000000, "d": 128, "K": 500,
         "nq": 10000, "m": 5, "m_to": 5, "ef": 200, "ef_to": 200},
        # the same loop on pinned host buffers with the learned budget
        {"name": "learned-d96", "kind": "search", "form": "learned", "call": "plan-host", "n": 200000, "d": 96,
         "K": 200, "nq": 4000, "m": 8, "m_to": 8, "ef": 200, "ef_to": 200},
        # a test-sized index built from nothing
        {"name": "build-3k-d64", "kind": "build", "n": 3001, "d": 64, "K": 40, "efc": 200, "iters": 5},
        # the same at a width that is no multiple of 16
        {"name": "build-5k-d100", "kind": "build", "n": 5000, "d": 100, "K": 40, "efc": 200, "iters": 5},
        # the CPU-runnable configuration of the benchmark
        {"name": "build-100k-d128", "kind": "build", "n": 100000, "d": 128, "K": 100, "efc": 400, "iters": 10},
        # build, then dynamic inserts into the built index, then the flat reverse lists
        {"name": "dynamic-30k-d96", "kind": "dynamic", "n": 20000, "more": 10000, "d": 96, "K": 64, "efc": 200,
         "iters": 5, "m_update": 10},
        # one gradient evaluation of the budget network (backward direction)
        {"name": "budget-gradients", "kind": "gradients", "n": 4096},
        # reverse lists of a KNN graph the caller owns, on the device
        {"name": "transpose-200k", "kind": "transpose", "n": 200000, "K": 100},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search"] * 6 + ["build"] * 2 + ["dynamic", "gradients", "transpose"])
    if kind == "gradients":
        return {"kind": kind, "n": _log(rng, 65, 4096)}
    if kind == "transpose":
        return {"kind": kind, "n": _log(rng, 1000, 200000), "K": _log(rng, 10, 100)}
    if kind == "build":
        d = rng.choice([32, 64, 96, 100, 128, 256])
        return {"kind": kind, "n": _log(rng, 1000, 6000 if d % 16 else 40000), "d": d, "K": rng.randint(20, 100),
                "efc": rng.choice([100, 200, 400]), "iters": rng.randint(3, 10)}
    if kind == "dynamic":
        n = _log(rng, 2000, 20000)
        return {"kind": kind, "n": n, "more": rng.randint(n // 8, n // 2), "d": rng.choice([32, 64, 96, 128]),
                "K": rng.randint(20, 64), "efc": rng.choice([100, 200]), "iters": rng.randint(3, 5),
                "m_update": rng.choice([0, 5, 10])}
    form = rng.choice(["exact", "exact", "bf16", "int8", "int8", "learned"])
    d = rng.choice([96, 128, 256] if form in ("bf16", "int8") else [96, 128] if form == "learned"
                   else [64, 96, 100, 128, 256])
    nq = _log(rng, 1, 10000)
    call = rng.choice(["plan", "plan-host"] if form == "learned" else ["host", "device", "plan", "plan-host"])
    m, ef = rng.randint(1, 10), rng.randint(50, 200)
    uneven = rng.random() < 0.4
    return {"kind": kind, "form": form, "call": call, "n": _log(rng, 2000, 10000 if d % 16 else 100000), "d": d,
            "K": rng.randint(20, 200), "nq": nq, "m": m, "m_to": rng.randint(m, 50) if uneven else m, "ef": ef,
            "ef_to": rng.randint(ef, 400) if uneven else ef}


def _mixture(n, d, components, centre_seed, draw_seed):
    g = torch.Generator(device="cuda").manual_seed(centre_seed)
    centres = 2.0 * torch.randn(components, d, generator=g, device="cuda")
    g.manual_seed(draw_seed)
    which = torch.randint(components, (n,), generator=g, device="cuda")
    return centres[which] + torch.randn(n, d, generator=g, device="cuda")


def _components(n):
    return max(8, min(256, n // 1500))


def _build(X, K, efc, iters, room=0):
    h = H.HRNN(X.shape[1], X.shape[0] + room, M, efc, 100, K)
    h.add_points(X)
    h.refineKNNG(iters, SAMPLE)
    return h


_indexes = {}  # the served indexes of this process, a few at a time
_stream = None


def _index(case):
    key = (case["n"], case["d"], case["K"], case["form"])
    h = _indexes.pop(key, None)
    if h is None:
        while len(_indexes) >= 2:
            _indexes.pop(next(iter(_indexes)))
        n, d = case["n"], case["d"]
        h = _build(_mixture(n, d, _components(n), 1000 + d, 7).cpu().numpy(), case["K"], EFC, 5)
        h.buildRKNNG()
        h.set_precision({"exact": H.PREC_FP32_EXACT, "bf16": H.PREC_BF16}.get(case["form"], H.PREC_INT8))
        if case["form"] == "learned":
            _give_budget(h, n, d)
    _indexes[key] = h
    return h


def _give_budget(h, n, d):
    """A network whose logits send a good part of the queries to each level (about
    40 % / 35 % / 25 %), with the features' own means and deviations as its
    normalisation; both kept to two digits."""
    def short(x):
        return np.array([float("%.1e" % v) for v in np.asarray(x, np.float64).ravel()], np.float32).reshape(np.shape(x))

    Q = _mixture(2000, d, _components(n), 1000 + d, 99).cpu().numpy()
    h.set_budget(False, 3, 8, 64, 0.9)
    f = h.budget_features(Q, NEAR, 8, 64)
    r = np.random.default_rng(5)
    p = [r.uniform(-1, 1, s).astype(np.float32) / np.float32(16) for s in H.BUDGET_SHAPES[:6]]
    sd = f.std(0)
    p += [short(f.mean(0)), short(np.where(sd > 1e-3, 1.0 / np.maximum(sd, 1e-3), 0.0))]
    h.budget_set_weights(p)
    z = h.budget_predict(f)
    for j, up in enumerate((1.5, 3.0)):
        scale = float("%.1e" % (3.0 / z[:, j].std()))
        p[4][j] *= np.float32(scale)
        p[5][j] = p[5][j] * np.float32(scale) + np.float32("%.1e" % (up - scale * z[:, j].mean()))
    h.budget_set_weights(p)
    h.set_budget(True, 3, 8, 64, 0.9)


def prepare(case, seed):
    global _stream
    kind = case["kind"]
    if kind in ("build", "dynamic"):
        n = case["n"] + case.get("more", 0)
        return dict(case, X=_mixture(n, case["d"], _components(n), seed, seed + 1).cpu().numpy())
    if kind == "gradients":
        r = np.random.default_rng(seed)
        h = H.HRNN(32, 16, 8, 32, 100, 8)
        p = [(r.uniform(-1, 1, s) / 16).astype(np.float32) for s in H.BUDGET_SHAPES[:6]]
        p += [np.zeros(256, np.float32), np.ones(256, np.float32)]
        h.budget_set_weights(p)
        X = r.standard_normal((case["n"], 256)).astype(np.float32)
        Y = (X @ r.standard_normal((256, 2)).astype(np.float32) > 0).astype(np.uint8)
        return dict(case, h=h, p=p, X=X, Y=Y)
    if kind == "transpose":
        n, K = case["n"], case["K"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        # K distinct other nodes per row, nearer ids more often, as in a clustered set
        step = 1 + torch.randint(max(1, (n - 1) // K), (n, K), generator=g, device="cuda")
        ids = (torch.arange(n, device="cuda")[:, None] + torch.cumsum(step, 1)) % n
        return dict(case, ids=ids.int(), cnt=torch.full((n,), K, dtype=torch.int32, device="cuda"),
                    off=torch.zeros(n + 1, dtype=torch.int64, device="cuda"),
                    ent=torch.zeros(n * K, dtype=torch.int32, device="cuda"))
    h, nq = _index(case), case["nq"]
    r = np.random.default_rng(seed)
    Q = _mixture(nq, case["d"], _components(case["n"]), 1000 + case["d"], 1000 + seed)
    m = r.integers(case["m"], case["m_to"] + 1, nq).astype(np.uint32)
    ef = r.integers(case["ef"], case["ef_to"] + 1, nq).astype(np.uint32)
    kp = np.full(nq, case["K"], np.uint32)
    state = dict(case, h=h, Q=Q.cpu().numpy(), mm=m, kp=kp, efs=ef, cap=max(1024, nq * 64))
    if case["call"] == "host":
        if nq > 1:
            state["out"] = [np.zeros(nq + 1, np.int64), np.zeros(state["cap"], np.int64)]
        return state
    state["dev"] = dict(Q=Q, m=torch.from_numpy(m.view(np.int32)).cuda(), kp=torch.from_numpy(kp.view(np.int32)).cuda(),
                        ef=torch.from_numpy(ef.view(np.int32)).cuda(),
                        off=torch.zeros(nq + 1, dtype=torch.int64, device="cuda"),
                        lab=torch.zeros(state["cap"], dtype=torch.int64, device="cuda"))
    t = state["dev"]
    if case["call"] == "device":
        return state
    if _stream is None:
        _stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    state["plan"] = h.search_plan(t["Q"].data_ptr(), nq, t["m"].data_ptr(), t["kp"].data_ptr(), t["ef"].data_ptr(),
                                  case["m_to"], case["ef_to"], 1.0, NEAR, t["off"].data_ptr(), t["lab"].data_ptr(),
                                  state["cap"], _stream.cuda_stream)
    if case["call"] == "plan-host":
        state["pin"] = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).pin_memory()
                        for a in (state["Q"], m, kp, ef)]
        state["pin"] += [torch.zeros(nq + 1, dtype=torch.int64).pin_memory(),
                         torch.zeros(state["cap"], dtype=torch.int64).pin_memory()]
    return state


def run(s):
    kind = s["kind"]
    if kind == "build":
        h = _build(s["X"], s["K"], s["efc"], s["iters"])
        h.buildRKNNG()
        off, ent = h.get_rknng()[:2]
        return {"offsets": off.view(np.int64), "entries": ent, "radius": h.get_kdist(min(NEAR, s["K"]))}
    if kind == "dynamic":
        n = s["n"]
        h = _build(s["X"][:n], s["K"], s["efc"], s["iters"], s["more"])
        h.buildRKNNG_mutable()
        h.insertPointDynamic(s["X"][n:], np.arange(n, n + s["more"], dtype=np.uint64), s["m_update"])
        h.buildRKNNG()
        off, ent = h.get_rknng()[:2]
        return {"offsets": off.view(np.int64), "entries": ent, "radius": h.get_kdist(min(NEAR, s["K"]))}
    if kind == "gradients":
        g, loss = s["h"].budget_gradients(s["X"], s["Y"])
        return {"grads": g, "loss": loss}
    if kind == "transpose":
        H.build_rknng_noalloc(s["ids"].data_ptr(), s["cnt"].data_ptr(), s["n"], s["K"], s["off"].data_ptr(),
                              s["ent"].data_ptr(), s["ent"].numel())
        return [s["off"], s["ent"]]
    h = s["h"]
    if s["call"] == "host":
        if s["nq"] == 1:
            got = h.searchRknn(s["Q"][0], s["m"], 1.0, NEAR, s["K"], s["ef"])
            return np.asarray(got + [-1] * (s["cap"] - len(got)), np.int64)
        off, lab = s["out"]
        h.search_rknn_batch_host(s["Q"].ctypes.data, s["nq"], s["mm"].ctypes.data, s["kp"].ctypes.data,
                                 s["efs"].ctypes.data, 1.0, NEAR, off.ctypes.data, lab.ctypes.data, s["cap"])
        return [off, lab]
    t = s["dev"]
    if s["call"] == "device":
        h.search_rknn_batch_device(t["Q"].data_ptr(), s["nq"], t["m"].data_ptr(), t["kp"].data_ptr(),
                                   t["ef"].data_ptr(), 1.0, NEAR, t["off"].data_ptr(), t["lab"].data_ptr(), s["cap"])
        return [t["off"], t["lab"]]
    if s["call"] == "plan":
        s["plan"].run(_stream.cuda_stream)
        return [t["off"], t["lab"]]
    q, m, kp, ef, off, lab = s["pin"]
    s["plan"].run_host(q.data_ptr(), m.data_ptr(), kp.data_ptr(), ef.data_ptr(), off.data_ptr(), lab.data_ptr(),
                       s["cap"], _stream.cuda_stream)
    return [off, lab]


def work(case):
    """Bytes and operations of one pass: a search scores about ten rows per beam
    entry and decides about 1.5 postings per reverse-list place of its proxies (rows
    at the form's bytes per element); a build scores about ten rows per
    construction beam entry and joins its samples about three times over."""
    kind, n, d = case["kind"], case["n"], case.get("d", 0)
    if kind == "gradients":
        return {"bytes": n * 1026 + 2 * 4 * H.BUDGET_PARAMS, "flops": 3 * 2 * n * (256 * 256 * 2 + 512)}
    if kind == "transpose":
        return {"bytes": 8 * n * case["K"] + 12 * n, "flops": 0}
    if kind in ("build", "dynamic"):
        n += case.get("more", 0)
        rows = n * (10 * case["efc"] + 3 * 1.5 * (2 * SAMPLE) ** 2)
        return {"bytes": n * (4 * d + 8 * case["K"] + 4 * case["K"]), "flops": 3.0 * d * rows}
    row = d * {"exact": 4, "bf16": 2}.get(case["form"], 1)
    m, ef = (case["m"] + case["m_to"]) / 2, (case["ef"] + case["ef_to"]) / 2
    rows = 10 * ef + 1.5 * m * case["K"]
    return {"bytes": case["nq"] * (rows * (row + 4) + 4 * d), "flops": 3.0 * d * case["nq"] * rows}


def exact(case, seed):
    """Only the gradients are computed numbers (searches and builds return ids and,
    from a build, distances between the neighbours that it found; the loss is a sum
    in no fixed order)."""
    if case["kind"] != "gradients":
        return None
    s = prepare(case, seed)
    W1, b1, W2, b2, W3, b3 = (torch.from_numpy(a).double().cuda().requires_grad_() for a in s["p"][:6])
    X, Y = torch.from_numpy(s["X"]).double().cuda(), torch.from_numpy(s["Y"]).double().cuda()
    gelu = torch.nn.functional.gelu
    z = gelu(gelu(X @ W1.T + b1) @ W2.T + b2) @ W3.T + b3
    loss = torch.nn.functional.binary_cross_entropy_with_logits(z, Y, reduction="sum") / case["n"]
    loss.backward()
    return {"grads": [w.grad for w in (W1, b1, W2, b2, W3, b3)], "loss": None}
