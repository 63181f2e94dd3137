"""The performance cases of the framework: what its users have it do, over the real range of sizes.

A case is a plain dict; `kind` says which public path it takes:
  step      grow_epoch + last_epoch_edges per cycle, from a checkpoint (the abm driver's loop)
  pa        run_epochs_out over several preferential-attachment epochs, from a checkpoint
  load      load_graph from host arrays, then run_epochs_out: a program's one pass over new inputs
  ensemble  the batched replicas: run_epochs_out over all of them, from a checkpoint
  er        run_er_epochs and the edges' copy-out, from a checkpoint
  er_out    pg_er_generate_noalloc into device buffers of the caller
  refcompat the reference's own per-paper model: run_epochs and the edges' copy-out, from a checkpoint
  lik       loglik + loglik_grad of a loaded growth trace at a batch of parameter points
  text      the grown graph's edge list and attribute rows as text
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from paragraph_gb300 import (PG_OK, PG_SAMPLER_ENUMERATE, PG_SAMPLER_THINNING, PG_WEIGHTS_REFCOMPAT, GrowthEngine,
                             PAParams, RCParams, ReplicaInput, TraceInput, _AttrRows, load_library)


def listed():
    return [
        # one small cycle of the abm driver: every launch and synchronisation counts
        {"name": "step_small", "kind": "step", "n": 2000, "cites": 10, "epochs": 1, "growth": 0.2, "degree": 15.0},
        # the plain configuration: 10,000 papers, 3 epochs of 5,000 new ones
        {"name": "pa_plain", "kind": "pa", "n": 10_000, "cites": 10, "pareto": False, "epochs": 3, "new": 5000,
         "growth": 0.0, "degree": 15.0, "enumerate": False},
        # the headline: a million papers with power-law in-degrees, 30 epochs at 3 % growth
        {"name": "pa_scale", "kind": "pa", "n": 1_000_000, "cites": 16, "pareto": True, "epochs": 30, "new": 0,
         "growth": 0.03, "degree": 30.0, "enumerate": False},
        # the other sampler, which enumerates each paper's 2-hop ball
        {"name": "pa_enumerate", "kind": "pa", "n": 30_011, "cites": 10, "pareto": False, "epochs": 3, "new": 0,
         "growth": 0.05, "degree": 20.0, "enumerate": True},
        # one run of a program from its input arrays to the new citations, page-locked buffers
        {"name": "load_run", "kind": "load", "n": 400_000, "cites": 16, "pareto": True, "epochs": 3, "growth": 0.03,
         "degree": 30.0, "pinned": True},
        # the batched ensemble: parameter studies over hundreds of independent graphs
        {"name": "ensemble", "kind": "ensemble", "replicas": 256, "lo": 5000, "hi": 200_000, "epochs": 10,
         "growth": 0.03, "degree": 20.0},
        # Erdos-Renyi growth at the densest configured p
        {"name": "er_dense", "kind": "er", "n": 100_000, "epochs": 10, "new": 10_000, "p": 1e-3},
        # one sparse Erdos-Renyi epoch into buffers the caller owns, odd sizes
        {"name": "er_out", "kind": "er_out", "n": 100_003, "new": 1017, "p": 1e-4},
        # the reference's own model with its options as the driver sets them
        {"name": "refcompat", "kind": "refcompat", "n": 200_000, "cites": 10, "epochs": 10, "growth": 0.03,
         "same_year": 0.1, "bag_mean": 15.0, "fixed": False},
        # calibration: a batch of points of a long trace, value and gradient
        {"name": "lik_batch", "kind": "lik", "n": 200_000, "cites": 10, "epochs": 10, "growth": 0.03, "degree": 20.0,
         "points": 64, "exact": False},
        # the last steps of a calibration: few points, exact arithmetic
        {"name": "lik_exact", "kind": "lik", "n": 20_011, "cites": 10, "epochs": 10, "growth": 0.03, "degree": 20.0,
         "points": 8, "exact": True},
        # the driver's output files: edge list and attribute rows of a grown graph
        {"name": "text", "kind": "text", "n": 100_000, "cites": 10, "epochs": 3, "growth": 0.03, "degree": 20.0},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.999))))

    kind = rng.choice(["step", "pa", "pa", "load", "ensemble", "er", "er_out", "refcompat", "lik", "lik", "text"])
    if kind == "step":
        return {"kind": kind, "n": logint(500, 50_000), "cites": rng.randint(3, 16), "epochs": rng.randint(1, 3),
                "growth": rng.uniform(0.01, 0.3), "degree": rng.uniform(5.0, 40.0)}
    if kind == "pa":
        if rng.random() < 0.25:
            return {"kind": kind, "n": logint(2000, 30_000), "cites": rng.randint(3, 10), "pareto": False,
                    "epochs": rng.randint(1, 3), "new": 0, "growth": rng.uniform(0.01, 0.05),
                    "degree": rng.uniform(5.0, 20.0), "enumerate": True}
        fixed = rng.random() < 0.3
        n = logint(3000, 900_000)
        return {"kind": kind, "n": n, "cites": rng.randint(4, 16), "pareto": rng.random() < 0.5,
                "epochs": rng.randint(1, 25), "new": logint(50, max(60, n // 30)) if fixed else 0,
                "growth": 0.0 if fixed else rng.uniform(0.01, 0.03), "degree": rng.uniform(5.0, 60.0 if n < 100_000 else 30.0),
                "enumerate": False}
    if kind == "load":
        return {"kind": kind, "n": logint(2000, 400_000), "cites": rng.randint(4, 16), "pareto": rng.random() < 0.5,
                "epochs": rng.randint(1, 3), "growth": rng.uniform(0.005, 0.03), "degree": rng.uniform(10.0, 30.0),
                "pinned": rng.random() < 0.5}
    if kind == "ensemble":
        return {"kind": kind, "replicas": logint(4, 200), "lo": logint(1000, 5000), "hi": logint(10_000, 200_000),
                "epochs": rng.randint(2, 10), "growth": rng.uniform(0.01, 0.03), "degree": rng.uniform(10.0, 20.0)}
    if kind == "er":
        return {"kind": kind, "n": logint(1000, 100_000), "epochs": rng.randint(1, 10), "new": logint(100, 10_000),
                "p": 10.0 ** rng.uniform(-5.0, -3.0)}
    if kind == "er_out":
        return {"kind": kind, "n": logint(1000, 1_000_000), "new": logint(100, 10_000), "p": 10.0 ** rng.uniform(-5.0, -3.0)}
    if kind == "refcompat":
        return {"kind": kind, "n": logint(2000, 150_000), "cites": rng.randint(4, 10), "epochs": rng.randint(1, 10),
                "growth": rng.uniform(0.01, 0.03), "same_year": rng.choice([0.0, 0.1, 0.3]),
                "bag_mean": rng.uniform(5.0, 15.0), "fixed": rng.random() < 0.5}
    if kind == "lik":
        exact = rng.random() < 0.4
        return {"kind": kind, "n": logint(2000, 20_000 if exact else 100_000), "cites": rng.randint(4, 10),
                "epochs": rng.randint(1, 10), "growth": rng.uniform(0.01, 0.03), "degree": rng.uniform(5.0, 20.0),
                "points": rng.choice([1, 2, 5, 8, 16, 33, 64]), "exact": exact}
    return {"kind": kind, "n": logint(1000, 100_000), "cites": rng.randint(3, 10), "epochs": rng.randint(1, 3),
            "growth": rng.uniform(0.01, 0.03), "degree": rng.uniform(5.0, 20.0)}


# ---------------------------------------------------------------- inputs (made on the GPU, handed over as host arrays)
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _host(t, pinned=True):
    t = t.to("cpu")
    return (t.pin_memory() if pinned else t).numpy()


def _seed_edges(g, n, cites, pareto):
    """(src, dst) of a seed graph on the GPU: uniform citations of earlier papers, or Pareto(2.5) target
    in-degrees of mean `cites` wired from later papers.  Repeated pairs collapse when loaded."""
    ids = torch.arange(n, device="cuda", dtype=torch.int64)
    if not pareto:
        src = ids[1:].repeat_interleave(cites)
        dst = (torch.rand(src.numel(), device="cuda", dtype=torch.float64, generator=g) * src).long()
        return src.int(), dst.int()
    u = 1.0 - torch.rand(n, device="cuda", dtype=torch.float64, generator=g)
    later = n - 1 - ids
    target = torch.minimum((cites * 0.6 * u ** -0.4).long(), later)
    dst = ids.repeat_interleave(target)
    span = later.repeat_interleave(target)
    src = dst + 1 + (torch.rand(dst.numel(), device="cuda", dtype=torch.float64, generator=g) * span).long()
    return src.int(), dst.int()


def _seed_nodes(g, n, by_id):
    ids = torch.arange(n, device="cuda", dtype=torch.int64)
    pub = ids * 5 // n - 5 if by_id else torch.randint(-5, 0, (n,), device="cuda", generator=g)
    fit = torch.exp(torch.randn(n, device="cuda", generator=g))
    return pub.int(), fit


def _seed_graph(case, g, pareto=False, pinned=True):
    src, dst = _seed_edges(g, case["n"], case["cites"], pareto)
    pub, fit = _seed_nodes(g, case["n"], pareto)
    return [_host(t, pinned) for t in (pub, fit, src, dst)]


def _grown(n, case):
    for _ in range(case["epochs"]):
        n += math.ceil(n * case["growth"]) if case.get("growth", 0.0) > 0 else case["new"]
    return n


def _params(case, **more):
    return PAParams(mean_out_degree=case["degree"], growth_rate=case["growth"], fixed_new_nodes=case.get("new", 0), **more)


def _out_buffers(cap, pinned=True):
    """(sources, targets) for `cap` citations; entries past the ones written stay zero."""
    return tuple(torch.zeros(int(cap), dtype=torch.int32, pin_memory=pinned).numpy() for _ in range(2))


def _edge_room(agents, degree):
    mu = agents * (degree + 1.0)
    return int(mu + 8.0 * mu ** 0.5 + 4096)


def _thetas(g, points):
    u = torch.rand((points, 4), device="cuda", dtype=torch.float64, generator=g).cpu().numpy()
    return np.array([0.5, 2.0, 0.5, 1.0]) + u * np.array([1.0, 8.0, 1.5, 7.0])


def _expand(off, col, nodes, owner):
    """Rows of `nodes` concatenated, each entry with its node's owner."""
    cnt = off[nodes + 1] - off[nodes]
    own = owner.repeat_interleave(cnt)
    first = (off[nodes] - (cnt.cumsum(0) - cnt)).repeat_interleave(cnt)
    return col[first + torch.arange(own.numel(), device="cuda")], own


def _balls(off, col, anchors, n):
    """[agents, n] membership of the undirected 2-hop ball of each agent's anchors."""
    A = anchors.shape[0]
    ball = torch.zeros(A * n, dtype=torch.bool, device="cuda")
    own = torch.arange(A, device="cuda").repeat_interleave(anchors.shape[1])
    z = anchors.reshape(-1)
    ball[own * n + z] = True
    z, own = _expand(off, col, z, own)
    key = torch.unique(own * n + z)
    ball[key] = True
    own, z = torch.div(key, n, rounding_mode="floor"), key % n
    ends = (off[z + 1] - off[z]).cumsum(0)
    i = 0
    while i < z.numel():  # at most about 200M entries at a time
        at = int(ends[i - 1]) if i else 0
        j = max(i + 1, int(torch.searchsorted(ends, at + 200_000_000)))
        v, o = _expand(off, col, z[i:j], own[i:j])
        ball[o * n + v] = True
        i = j
    return ball.view(A, n)


def _undirected(src, dst, n):
    a, b = torch.cat([src, dst]).long(), torch.cat([dst, src]).long()
    key = torch.unique(a * n + b)
    rows = torch.div(key, n, rounding_mode="floor")
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.bincount(rows, minlength=n).cumsum(0)
    return off, key % n


def _trace(case, seed, keep=None):
    """A growth trace drawn with torch alone from the model at (1, 5, 1, 4): each paper's candidates come
    from the global weights and are kept if in the paper's ball or with probability 1/4, first come
    first.  keep(epoch, agents, ball, weights' inputs) sees the balls as they are made."""
    g = _gen(seed)
    n0, beta = case["n"], 4.0
    src, dst = _seed_edges(g, n0, case["cites"], False)
    pub, fit = _seed_nodes(g, n0, False)
    src0, dst0 = src, dst
    nodes, times, anchors, counts, cites = [n0], [], [], [], []
    for e in range(case["epochs"]):
        n = nodes[-1]
        A = math.ceil(n * case["growth"])
        off, col = _undirected(src, dst, n)
        key = torch.unique(src.long() * n + dst.long())
        indeg = torch.bincount(key % n, minlength=n)
        w = fit.double() * (indeg + 1.0) * torch.exp(-(e - pub.double()) / 5.0)
        cdf = w.cumsum(0)
        anc = (torch.rand((A, 3), device="cuda", dtype=torch.float64, generator=g) * n).long()
        k = torch.poisson(torch.full((A,), case["degree"], device="cuda"), generator=g).long().clamp(1, 64)
        new_src, new_dst = [], []
        for a0 in range(0, A, max(1, 400_000_000 // n)):
            a1 = min(A, a0 + max(1, 400_000_000 // n))
            ball = _balls(off, col, anc[a0:a1], n)
            cand = torch.searchsorted(cdf, torch.rand((a1 - a0, 512), device="cuda", dtype=torch.float64, generator=g)
                                      * cdf[-1], right=True).clamp_(max=n - 1)
            ok = ball.gather(1, cand) | (torch.rand(cand.shape, device="cuda", generator=g) < 1.0 / beta)
            order = torch.argsort(cand, dim=1, stable=True)  # repeats: only a node's first acceptance counts
            sc, so = cand.gather(1, order), ok.gather(1, order)
            cum = so.int().cumsum(1)
            head = torch.ones_like(so)
            head[:, 1:] = sc[:, 1:] != sc[:, :-1]
            before = torch.cummax(torch.where(head, cum - so.int(), -1), 1).values
            first = torch.zeros_like(ok).scatter_(1, order, so & (cum - so.int() == before))
            rank = first.int().cumsum(1)
            take = first & (rank <= k[a0:a1, None])
            counts.append(take.sum(1))
            row, at = torch.nonzero(take, as_tuple=True)
            new_src.append(row + a0 + n)
            new_dst.append(cand[row, at])
            if keep is not None:
                keep(e, a0, ball, fit, indeg, pub, n)
        src, dst = torch.cat([src.long()] + new_src), torch.cat([dst.long()] + new_dst)
        cites += new_dst
        anchors.append(torch.cat([anc, torch.full((A, 1), -1, device="cuda")], 1))
        times.append(e)
        nodes.append(n + A)
        pub = torch.cat([pub, torch.full((A,), e, device="cuda", dtype=torch.int32)])
        fit = torch.cat([fit, torch.exp(torch.randn(A, device="cuda", generator=g))])
    off = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), torch.cat(counts).cumsum(0)])
    theta = _thetas(g, case["points"])
    return dict(pub=pub, fitness=fit, seed_src=src0, seed_dst=dst0, epoch_nodes=np.array(nodes), epoch_t=np.array(times),
                anchors=torch.cat(anchors), cite_off=off, cites=torch.cat(cites)), theta


# ---------------------------------------------------------------- a case's state and one pass
def prepare(case, seed):
    kind = case["kind"]
    g = _gen(seed)
    st = {"kind": kind, "case": case}
    if kind in ("step", "pa"):
        enum = case.get("enumerate", False)
        eng = GrowthEngine(seed=seed, sampler=PG_SAMPLER_ENUMERATE if enum else PG_SAMPLER_THINNING)
        eng.load_graph(*_seed_graph(case, g, case.get("pareto", False)), _params(case), planned_epochs=case["epochs"])
        eng.checkpoint()
        st["out"] = _out_buffers(_edge_room(_grown(case["n"], case) - case["n"], case["degree"]))
        if kind == "step":
            st["out"] = [_out_buffers(_edge_room(_grown(case["n"], case), case["degree"])) for _ in range(case["epochs"])]
    elif kind == "load":
        eng = GrowthEngine(seed=seed)
        st["graph"] = _seed_graph(case, g, case["pareto"], case["pinned"])
        room = _edge_room(_grown(case["n"], case) - case["n"], case["degree"])
        st["out"] = _out_buffers(room, case["pinned"])
    elif kind == "ensemble":
        rng = np.random.Generator(np.random.PCG64(seed))
        # sizes spread evenly over the logarithm, so that every seed has the same amount of work
        steps = (np.arange(case["replicas"]) + 0.5) / case["replicas"]
        sizes = rng.permutation(case["lo"] * (case["hi"] / case["lo"]) ** steps).astype(int)
        reps, room = [], 4096
        for n in sizes:
            one = {"n": int(n), "cites": 10}
            prm = _params(case, alpha=float(rng.uniform(0.5, 1.5)), tau=float(rng.uniform(2, 10)),
                          gamma=float(rng.uniform(0.5, 2.0)), beta=float(rng.uniform(1, 8)))
            reps.append(ReplicaInput(*_seed_graph(one, g, pinned=False), prm, planned_epochs=case["epochs"]))
            room += _edge_room(_grown(int(n), case) - int(n), case["degree"])
        eng = GrowthEngine(seed=seed, replicas=case["replicas"])
        eng.load_replicas(reps)
        eng.checkpoint()
        st["out"] = _out_buffers(room)
    elif kind == "er":
        eng = GrowthEngine(seed=seed)
        n, room = case["n"], 0
        for _ in range(case["epochs"]):
            mu = case["new"] * n * case["p"]
            room += int(mu + 8 * mu ** 0.5 + 1024) + 1
            n += case["new"]
        eng.load_graph(np.full(case["n"], -1, np.int32), np.ones(case["n"], np.float32), np.zeros(0, np.int32),
                       np.zeros(0, np.int32), PAParams(), planned_epochs=1)
        eng.reserve(n, room)
        eng.checkpoint()
        st["out"] = _out_buffers(room)
    elif kind == "er_out":
        mu = case["new"] * case["n"] * case["p"]
        st["seed"] = seed
        st["lib"] = load_library()
        st["dev"] = torch.zeros((2, int(mu + 8 * mu ** 0.5 + 1024)), dtype=torch.int32, device="cuda")
        st["stream"] = torch.cuda.current_stream().cuda_stream
        return st
    elif kind == "refcompat":
        eng = GrowthEngine(seed=seed, weight_model=PG_WEIGHTS_REFCOMPAT)
        pub, fit, src, dst = _seed_graph(case, g)
        rng = np.random.Generator(np.random.PCG64(seed))
        v = np.arange(1, 1001, dtype=np.float64)
        fit = rng.choice(v, size=case["n"], p=v ** -1.634 / (v ** -1.634).sum()).astype(np.float32)
        pub = np.sort(rng.integers(-10, 0, size=case["n"])).astype(np.int32)
        bag = np.clip(rng.poisson(case["bag_mean"], size=1000), 0, 300).astype(np.int32)
        rec = 0.8 ** np.arange(40.0)
        eng.load_graph(pub, fit, src, dst, PAParams(growth_rate=case["growth"]), planned_epochs=case["epochs"])
        mix = dict(pa_weight=0.5, rec_weight=0.3, fit_weight=0.2, alpha=0.6) if case["fixed"] else {}
        eng.rc_configure(RCParams(growth_rate=case["growth"], same_year=case["same_year"], **mix), bag, rec / rec.sum())
        n0, m0 = eng.counts()
        n1 = _grown(n0, case)
        eng.reserve(n1, m0 + (n1 - n0) * int(min(bag.max(), 256)))
        eng.checkpoint()
        st["out"] = _out_buffers(_edge_room(n1 - n0, 2.0 * case["bag_mean"]))
    elif kind == "lik":
        eng = GrowthEngine(seed=seed)
        t, st["theta"] = _trace(case, seed)
        eng.load_trace(TraceInput(**{k: v.cpu().numpy() if isinstance(v, torch.Tensor) else v for k, v in t.items()}))
        eng.set_lik_exact_exp2(case["exact"])
        del t
        torch.cuda.empty_cache()
    else:
        eng = GrowthEngine(seed=seed)
        eng.load_graph(*_seed_graph(case, g), _params(case), planned_epochs=case["epochs"])
        eng.run_epochs(case["epochs"])
        n, _ = eng.counts()
        rng = np.random.Generator(np.random.PCG64(seed))
        st["ids"] = np.sort(rng.choice(50 * n, size=n, replace=False)).astype(np.int64)
        st["draws"] = rng.random((n, 4))
        st["draws"][:case["n"]] = -1.0
        st["ints"] = rng.integers(0, 1000, size=(n, 4)).astype(np.int32)
        st["gens"] = np.where(rng.random((n, 4)) < 0.25, -1, st["ids"][rng.integers(0, n, size=(n, 4))])
        m = case["n"] * case["cites"] + _edge_room(n - case["n"], case["degree"])
        st["text"] = np.zeros(20 * m, np.uint8), np.zeros(200 * n, np.uint8)
    st["eng"] = eng
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "er_out":
        ne = ctypes.c_int64()
        src, dst = st["dev"]
        rc = st["lib"].pg_er_generate_noalloc(st["seed"], 3, case["n"], case["new"], case["p"], src.data_ptr(),
                                              dst.data_ptr(), src.numel(), ctypes.byref(ne), st["stream"])
        if rc != PG_OK:
            raise RuntimeError("pg_er_generate_noalloc: status %d" % rc)
        return src, dst, ne.value
    eng = st["eng"]
    if kind == "lik":
        return eng.loglik(st["theta"]), eng.loglik_grad(st["theta"])
    if kind == "text":
        # as the driver writes its files, through the C interface: the size, then the text
        lib, ctx, ids, size = eng._lib, eng._ctx, st["ids"], ctypes.c_int64()
        rows = _AttrRows(len(ids), case["n"], ids.ctypes.data, st["draws"].ctypes.data, st["ints"].ctypes.data,
                         st["gens"].ctypes.data, 0, 0)
        sizes = []
        for buf, fmt in zip(st["text"], (lambda *a: lib.pg_format_edges(ctx, 0, ids.ctypes.data, len(ids), *a),
                                         lambda *a: lib.pg_format_attributes(ctx, 0, ctypes.byref(rows), *a))):
            if fmt(None, 0, ctypes.byref(size)) != PG_OK or size.value > len(buf):
                raise RuntimeError("text size")
            if fmt(buf.ctypes.data, size.value, ctypes.byref(size)) != PG_OK:
                raise RuntimeError("text")
            sizes.append(size.value)
        return st["text"], sizes
    if kind == "load":
        eng.load_graph(*st["graph"], _params(case), planned_epochs=case["epochs"])
        eng.set_epoch(0)
        return st["out"], eng.run_epochs_out(case["epochs"], st["out"], use_graph=False)
    eng.restore()
    if kind == "step":
        sizes = []
        for e in range(case["epochs"]):
            sizes.append(eng.grow_epoch())
            first, count = eng.epoch_edges()
            eng.edges(first, count, out=st["out"][e])
        return st["out"], sizes
    if kind == "er":
        ne = eng.run_er_epochs(case["epochs"], case["new"], case["p"])
        eng.edges(0, ne, out=st["out"])
        return st["out"], ne
    if kind == "refcompat":
        _, m0 = eng.counts()
        ne = eng.run_epochs(case["epochs"])
        eng.edges(m0, ne, out=st["out"])
        return st["out"], ne
    return st["out"], eng.run_epochs_out(case["epochs"], st["out"])


# ---------------------------------------------------------------- the work of a pass
def work(case):
    """Bytes: the seed graph's arrays read once, the new citations written once (as pairs).  Operations:
    a weight per node and epoch (20 each), a draw per citation (100); for the likelihood the weights and
    sums of every ball element and point, with balls of about anchors * (2 * mean degree)^2 papers."""
    kind = case["kind"]
    if kind in ("er", "er_out"):
        n, edges = case["n"], 0.0
        for _ in range(case.get("epochs", 1)):
            edges += case["new"] * n * case["p"]
            n += case["new"]
        return {"bytes": 8.0 * edges + 8.0 * n, "flops": 100.0 * edges}
    if kind == "ensemble":
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"]) if case["hi"] > case["lo"] else case["hi"]
        n0, n1, reps, degree = mean, mean * (1 + case["growth"]) ** case["epochs"], case["replicas"], case["degree"]
        cites = 10
    else:
        n0, n1, reps, cites = case["n"], _grown(case["n"], case), 1, case["cites"]
        degree = case.get("degree", case.get("bag_mean"))
    new = (n1 - n0) * degree
    if kind == "lik":
        ball = min(n0, 3.0 * (2.0 * cites) ** 2)
        return {"bytes": 8.0 * n1 + 4.0 * n0 * cites + 4.0 * new + 12.0 * (n1 - n0),
                "flops": 20.0 * case["points"] * (2.0 * case["epochs"] * n0 + (n1 - n0) * (ball + degree))}
    if kind == "text":
        return {"bytes": 12.0 * (n0 * cites + new) + 16.0 * (n0 * cites + new) + 100.0 * n1 + 88.0 * n1, "flops": 0.0}
    return {"bytes": reps * (8.0 * n1 + 8.0 * n0 * cites + 8.0 * new),
            "flops": reps * (20.0 * n0 * case["epochs"] + 100.0 * new)}


# ---------------------------------------------------------------- the likelihood in 64 bits
def exact(case, seed):
    """log L and its gradient at every point, in 64 bits: Z_a and its derivatives as a sum over all papers
    plus (beta - 1) times the sum over the agent's ball, then the citations in draw order.  The other
    kinds return whole numbers."""
    if case["kind"] != "lik":
        return None
    seen = []

    def keep(e, a0, ball, fit, indeg, pub, n):
        rows = ball.sum(1)
        seen.append((e, torch.nonzero(ball.view(-1)).view(-1).remainder_(n).int(), rows, fit[:n], indeg, pub[:n], n))

    t, theta = _trace(case, seed, keep)
    off, cites = t["cite_off"], t["cites"]
    th = torch.from_numpy(theta).cuda()
    B = th.shape[0]
    ll = torch.zeros(B, dtype=torch.float64, device="cuda")
    grad = torch.zeros((B, 4), dtype=torch.float64, device="cuda")
    a = 0
    for e, ids, rows, fit, indeg, pub, n in seen:
        A = rows.numel()
        x = torch.stack([torch.log(indeg + 1.0), e - pub.double(), torch.log(fit.double())], 1)  # [n, 3]
        c0, c1 = int(off[a]), int(off[a + A])
        k = (off[a + 1:a + A + 1] - off[a:a + A])
        own = torch.arange(A, device="cuda").repeat_interleave(k)
        cid = cites[c0:c1]
        lo = rows.cumsum(0) - rows
        where = torch.repeat_interleave(torch.arange(A, device="cuda"), rows) * n + ids
        pos = torch.searchsorted(where, own * n + cid).clamp_(max=max(0, where.numel() - 1))
        inball = where[pos] == own * n + cid
        del where, pos
        start = (off[a:a + A] - c0).clamp(max=max(0, c1 - c0 - 1))
        w = torch.exp(x[:, 2:] * th[:, 2] + x[:, :1] * th[:, 0] - x[:, 1:2] / th[:, 1])  # [n, B]
        d = torch.stack([x[:, :1].expand(n, B), x[:, 1:2] / (th[:, 1] ** 2), x[:, 2:].expand(n, B)], 2)  # d log w
        wd = torch.cat([w[:, :, None], w[:, :, None] * d], 2)  # [n, B, 4]
        crow = torch.cat([lo[:1] * 0, rows.cumsum(0)])
        inc = torch.sparse_csr_tensor(crow, ids.long(), torch.ones(ids.numel(), dtype=torch.float64, device="cuda"), (A, n))
        bsum = (inc @ wd.view(n, 4 * B)).view(A, B, 4)
        z = torch.cat([wd.sum(0) + (th[:, 3:] - 1.0) * bsum, bsum[:, :, :1]], 2)  # Z, dZ by alpha, tau, gamma, beta
        wc = wd[cid] * torch.where(inball[:, None], th[:, 3], 1.0)[:, :, None]
        cols = torch.cat([wc, (w[cid] * inball[:, None])[:, :, None]], 2)
        cum = cols.cumsum(0) - cols  # drawn before
        rest = (z + (cum[start] if c1 > c0 else 0.0)).repeat_interleave(k, 0) - cum
        ll += (torch.log(wc[:, :, 0]) - torch.log(rest[:, :, 0])).sum(0)
        own_d = torch.cat([d[cid], (inball[:, None] / th[:, 3])[:, :, None]], 2)
        grad += (own_d - rest[:, :, 1:] / rest[:, :, :1]).sum(0)
        a += A
    return ll, grad
