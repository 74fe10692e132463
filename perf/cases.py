"""What the framework is timed on: its public entry points over their real range.

A case is a dict: `kind` names the entry point, the rest are sizes and options.

  points   f2m_solve_points, one instance: `shape` is "uniform" (integer
           coordinates in a 10^4 box, the small and medium single solves),
           "lattice" (a 30% filled integer lattice, the tie-rich geometry of
           the VLSI instances, whose combs need Ax=b and at times the repair
           loop) or "clustered" (Gaussian clusters and 10% background, the
           large-instance configuration)
  knn      f2m_knn, the candidate graph alone (3-decimal coordinates)
  batch    many independent instances in one call, sizes log-uniform in
           [lo, hi]: Context.solve_batch from host arrays, or
           solve_batch_device with `resident` inputs and outputs; `nint`
           switches to TSPLIB's rounded costs
  smooth   Context.smoothed_bound, the differentiable bound: `count`
           jittered-lattice instances of lo..hi points, or with count = 1 one
           uniform instance; forward alone or with the coordinate gradient

The single-instance results go into arrays of the caller's, sized for the
most edges the call can return (n * top_k; the rest stays zero), through the
C ABI as Context does it.

`exact` restates what has a value of its own in plain FP64 torch: the LP
value (any convergent dual ascent reaches it), the candidate graph's costs,
and the smoothed bound with its adjoint.
"""
import ctypes
import math
import time

import numpy as np
import torch

import f2m_b200
from f2m_b200 import synth


def listed():
    return [
        # latency of one small solve: the smoke instance and the 1,000-point configuration
        dict(name="points_300", kind="points", shape="uniform", n=300, top_k=12),
        dict(name="points_1000", kind="points", shape="uniform", n=1000, top_k=20),
        # the largest sizes of the batched configuration, solved one at a time
        dict(name="points_5000", kind="points", shape="uniform", n=5000, top_k=16),
        # VLSI geometry: equal distances, half-integral combs
        dict(name="lattice_1500", kind="points", shape="lattice", n=1500, top_k=12),
        # large single instances, the headline use of the reference
        dict(name="clustered_20k", kind="points", shape="clustered", n=20000, top_k=16),
        dict(name="clustered_100k", kind="points", shape="clustered", n=100000, top_k=50),
        # the graph alone, for callers with a solver of their own
        dict(name="knn_20k", kind="knn", n=20000, top_k=24),
        # a small batch of small instances with integer costs, from host arrays
        dict(name="batch_64", kind="batch", count=64, lo=50, hi=320, top_k=10, nint=True, resident=False),
        # the batched configuration, resident in device memory
        dict(name="batch_4096", kind="batch", count=4096, lo=50, hi=5000, top_k=16, nint=False, resident=True),
        # evaluating the smoothed bound of a few instances at a milder temperature
        dict(name="smooth_fwd_24", kind="smooth", count=24, lo=200, hi=600, top_k=24, tau=1e-2, iters=40, grad=False),
        # the two differentiated configurations: many instances, one large instance
        dict(name="smooth_1024", kind="smooth", count=1024, lo=200, hi=2000, top_k=24, tau=1e-3, iters=100, grad=True),
        dict(name="smooth_10k", kind="smooth", count=1, lo=10000, hi=10000, top_k=30, tau=1e-3, iters=100, grad=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["points", "points", "clustered", "knn", "batch", "batch", "smooth", "smooth"])
    if kind == "points":
        return dict(kind="points", shape="uniform", n=_log_int(rng, 100, 9000), top_k=rng.randint(8, 24))
    if kind == "clustered":
        return dict(kind="points", shape="clustered", n=_log_int(rng, 10500, 80000), top_k=rng.randint(10, 40))
    if kind == "knn":
        return dict(kind="knn", n=_log_int(rng, 500, 80000), top_k=rng.randint(5, 40))
    if kind == "batch":
        return dict(kind="batch", count=_log_int(rng, 8, 1500), lo=rng.randint(30, 90), hi=_log_int(rng, 200, 4000),
                    top_k=rng.randint(8, 24), nint=rng.random() < 0.3, resident=rng.random() < 0.5)
    case = dict(kind="smooth", count=1, lo=0, hi=0, top_k=rng.randint(8, 32), tau=rng.choice([1e-3, 1e-2, 5e-2]),
                iters=rng.randint(20, 100), grad=rng.random() < 0.7)
    if rng.random() < 0.4:
        case["lo"] = case["hi"] = _log_int(rng, 200, 10000)
    else:
        case["count"] = _log_int(rng, 8, 800)
        case["lo"] = rng.randint(50, 300)
        case["hi"] = _log_int(rng, 400, 2000)
    return case


def _inputs(case, seed):
    """(offs, x, y) of the case, host arrays."""
    kind = case["kind"]
    if kind == "batch" or case.get("count", 1) > 1:  # sizes by the case, points by the seed
        count, lo, hi = case["count"], case["lo"], case["hi"]
        if kind == "batch":
            sizes = synth.batch_sizes(count, 3, lo, hi)
        else:
            sizes = lo + np.floor(synth.uniform(5, 320, count) * (hi - lo + 1)).astype(np.int64)
        offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
        if kind == "batch":
            x, y = synth.uniform_int_points(int(offs[-1]), seed)
        else:
            parts = [synth.jittered_lattice(int(m), seed * 100_000 + b) for b, m in enumerate(sizes)]
            x, y = (np.concatenate(p) for p in zip(*parts))
        return offs, x, y
    n = case["hi"] if kind == "smooth" else case["n"]
    if kind == "smooth":
        x, y = synth.config4(seed, n)
    elif kind == "knn":
        x, y = (np.floor(synth.uniform(seed, s, n) * 1e7) / 1e3 for s in (0, 1))
    elif case["shape"] == "uniform":
        x, y = synth.uniform_int_points(n, seed)
    elif case["shape"] == "lattice":
        x, y = synth.lattice_points(n, seed, keep=0.3)
    else:
        x, y = synth.config2(seed, n=n)
    return np.array([0, n], np.int64), x, y


def prepare(case, seed):
    offs, x, y = _inputs(case, seed)
    state = dict(case=case, ctx=f2m_b200.default_context(), offs=offs, x=x, y=y)
    if case["kind"] == "smooth":
        state["params"] = f2m_b200.default_smooth_params(tau=case["tau"], iters=case["iters"])
    elif case["kind"] == "batch":
        mode = f2m_b200.COST_NINT if case["nint"] else f2m_b200.COST_REF_EUCLID
        state["params"] = f2m_b200.default_params(cost_mode=mode)
        if case["resident"]:
            n = case["count"]
            state["device"] = [torch.from_numpy(a).cuda() for a in (offs, x, y)]
            state["lp"] = torch.empty(n, dtype=torch.float64, device="cuda")
            state["status"] = torch.empty(n, dtype=torch.int32, device="cuda")
            state["iterations"] = torch.empty(n, dtype=torch.int64, device="cuda")
    else:
        state["params"] = f2m_b200.default_params()
        n, cap = case["n"], case["n"] * case["top_k"]
        state["edges"] = {k: np.zeros(cap, t) for k, t in (
            ("v1", np.int32), ("v2", np.int32), ("lab1", np.int32), ("lab2", np.int32),
            ("Do", np.float64), ("D", np.float64), ("x", np.float64))}
        state["nodes"] = {"label": np.zeros(n, np.int32), "F": np.zeros(n, np.float64)}
    return state


def _ptr(a):
    return ctypes.c_void_p(a.ctypes.data)


def _single(state, knn):
    """One call of f2m_solve_points or f2m_knn with its results fetched."""
    case, L, h = state["case"], f2m_b200.lib(), ctypes.c_void_p()
    x, y, n, k = _ptr(state["x"]), _ptr(state["y"]), case["n"], case["top_k"]
    if knn:
        status = L.f2m_knn(state["ctx"].handle, x, y, None, n, k, ctypes.byref(h))
    else:
        status = L.f2m_solve_points(state["ctx"].handle, x, y, None, n, k, ctypes.byref(state["params"]),
                                    ctypes.byref(h))
    if not h:
        raise f2m_b200.F2MError(status, state["ctx"].last_error())
    out = {"status": status, "n_nodes": L.f2m_result_n_nodes(h), "n_edges": L.f2m_result_n_edges(h)}
    edges, nodes = state["edges"], state["nodes"]
    L.f2m_result_edges(h, *(_ptr(a) for a in edges.values()))
    L.f2m_result_nodes(h, *(_ptr(a) for a in nodes.values()))
    if not knn:
        stats = f2m_b200.Stats()
        L.f2m_result_stats(h, ctypes.byref(stats))
        out.update(lp=L.f2m_result_lp(h), max_rank=L.f2m_result_max_rank(h), iterations=stats.iterations)
    L.f2m_result_free(h)
    out.update(edges, **nodes)
    return out


def run(state):
    case, ctx = state["case"], state["ctx"]
    if case["kind"] == "smooth":
        if not case["grad"]:
            return {"L": ctx.smoothed_bound(state["offs"], state["x"], state["y"], case["top_k"], state["params"])}
        L, gx, gy = ctx.smoothed_bound(state["offs"], state["x"], state["y"], case["top_k"], state["params"], grad=True)
        return {"L": L, "gx": gx, "gy": gy}
    if case["kind"] == "batch":
        if not case["resident"]:
            return ctx.solve_batch(state["offs"], state["x"], state["y"], case["top_k"], state["params"], details=True)
        offs, x, y = (t.data_ptr() for t in state["device"])
        ctx.solve_batch_device(state["offs"], offs, x, y, case["top_k"], state["lp"].data_ptr(),
                               state["status"].data_ptr(), state["params"], state["iterations"].data_ptr())
        return {k: state[k] for k in ("lp", "status", "iterations")}
    return _single(state, case["kind"] == "knn")


def _mean_size(case):
    if case["kind"] == "batch":  # log-uniform
        return (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
    return (case["lo"] + case["hi"]) / 2


def work(case):
    """Points in, results out; the arithmetic of the sweeps over the lists.

    The union of the N nearest holds about 0.6 N edges a point.  A solve
    sweeps about four active entries a node (two additions and three compares
    each) over a thousand steps at the least; a step of the smoothed bound
    takes about 16 operations for each of the few list entries within reach of
    the root, twice for the forward pass and three times more for the adjoint."""
    if case["kind"] == "smooth":
        n = case["count"] * _mean_size(case)
        passes = 5 if case["grad"] else 1
        return {"bytes": n * (8 + (8 if case["grad"] else 0)) + 16 * case["count"],
                "flops": n * case["iters"] * passes * 4 * 16}
    if case["kind"] == "batch":
        n = case["count"] * _mean_size(case)
        return {"bytes": 16 * n + 28 * case["count"], "flops": n * 1000 * 4 * 5}
    n, edges = case["n"], 0.6 * case["n"] * case["top_k"]
    if case["kind"] == "knn":
        return {"bytes": 16 * n + 24 * edges + 4 * n, "flops": n * 3 * case["top_k"] * 5}
    return {"bytes": 16 * n + 40 * edges + 12 * n, "flops": n * 1000 * 4 * 5}


# -- the same values in plain FP64 torch ------------------------------------

_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _union_pairs(x, y, top_k, dist):
    """Pairs a < b where one is among the other's top_k nearest (ties by index)."""
    n = len(x)
    k = min(top_k, n - 1)
    a, b = [], []
    step = max(1, (1 << 25) // n)
    for s in range(0, n, step):
        d = dist(x[s:s + step, None], y[s:s + step, None], x[None], y[None])
        m = d.shape[0]
        d[torch.arange(m, device=_DEV), torch.arange(s, s + m, device=_DEV)] = math.inf
        if d.dtype == torch.float32:  # order by (cost, index)
            key = (d.view(torch.int32).long() << 32) | torch.arange(n, device=_DEV)
            near = torch.topk(key, k, dim=1, largest=False).indices
        else:
            near = torch.topk(d, k, dim=1, largest=False).indices
        me = torch.arange(s, s + m, device=_DEV)[:, None].expand_as(near)
        a.append(torch.minimum(me, near).reshape(-1))
        b.append(torch.maximum(me, near).reshape(-1))
    code = torch.unique(torch.cat(a) * n + torch.cat(b))
    return code // n, code % n


def _padded(a, b, n):
    """(nbr, slot) [n, max degree]: neighbours and edge of each list entry (edge len(a): padding)."""
    v, w = torch.cat([a, b]), torch.cat([b, a])
    e = torch.arange(len(a), device=_DEV).repeat(2)
    order = torch.argsort(v * n + w)
    v, w, e = v[order], w[order], e[order]
    deg = torch.bincount(v, minlength=n)
    pos = torch.arange(len(v), device=_DEV) - (torch.cumsum(deg, 0) - deg)[v]
    nbr = torch.zeros(n, int(deg.max()), dtype=torch.long, device=_DEV)
    edge = torch.full_like(nbr, len(a))
    nbr[v, pos] = w
    edge[v, pos] = e
    return nbr, edge


def _dist64(x0, y0, x1, y1):
    return torch.sqrt((x0 - x1) ** 2 + (y0 - y1) ** 2)


def _dist32(x0, y0, x1, y1):
    """The FP32 distance, every operation rounded once (the root through FP64)."""
    dx, dy = x0 - x1, y0 - y1
    return torch.sqrt((dx * dx + dy * dy).double()).float()


def _exact_lp(case, offs, x, y):
    """The LP value of each instance by Jacobi dual ascent over the whole lists, or None when it takes too long."""
    began = time.monotonic()
    a_all, b_all, c_all, inst, base = [], [], [], [], 0
    for i in range(len(offs) - 1):
        p = np.unique(np.stack([x[offs[i]:offs[i + 1]], y[offs[i]:offs[i + 1]]]), axis=1)
        px, py = (torch.from_numpy(q).to(_DEV) for q in p)
        a, b = _union_pairs(px, py, case["top_k"], _dist64)
        c = _dist64(px[a], py[a], px[b], py[b])
        a_all.append(a + base)
        b_all.append(b + base)
        c_all.append(torch.floor(c + 0.5) if case.get("nint") else c)
        inst.append(torch.full((len(px),), i, device=_DEV))
        base += len(px)
    a, b, c, inst = (torch.cat(t) for t in (a_all, b_all, c_all, inst))
    nbr, edge = _padded(a, b, base)
    D = torch.cat([c, torch.tensor([math.inf], dtype=torch.float64, device=_DEV)])[edge]
    h = torch.zeros(base, dtype=torch.float64, device=_DEV)
    tol = 1e-11 * float(c.mean())
    for it in range(1, 60001):
        near = torch.topk(D + h[:, None] + h[nbr], 3, dim=1, largest=False, sorted=True).values
        g = -(near[:, 1] + near[:, 2]) / 4
        h = h + g
        if it % 200 == 0:
            if float(g.abs().max()) < tol:
                break
            if time.monotonic() - began > 15:
                return None
    else:
        return None
    val = torch.zeros(len(offs) - 1, dtype=torch.float64, device=_DEV)
    val.index_add_(0, inst, -2 * h)
    val.index_add_(0, inst[a], torch.clamp(c + h[a] + h[b], max=0.0))
    return val.cpu().numpy()


def _logit(z):
    """(sum sigma - 2, its scale, its slope) by rows, without cancellation."""
    e = torch.exp(-z.abs())
    m = e / (1 + e)
    up = z >= 0
    g = up.sum(1) - 2 + torch.where(up, -m, m).sum(1)
    return g, m.sum(1), (m / (1 + e)).sum(1)


def _exact_smooth(case, offs, x, y):
    tau, omega = case["tau"], 0.5
    fx, fy = (torch.from_numpy(q).to(_DEV) for q in (x, y))
    parts = []
    for i in range(len(offs) - 1):
        s, e = int(offs[i]), int(offs[i + 1])
        a, b = _union_pairs(fx[s:e], fy[s:e], case["top_k"], _dist32)
        parts.append((a + s, b + s))
    a, b = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
    n = len(x)
    ce = _dist32(fx[a], fy[a], fx[b], fy[b]).double()
    nbr, edge = _padded(a, b, n)
    c = torch.cat([ce, torch.tensor([math.inf], dtype=torch.float64, device=_DEV)])[edge]
    u = torch.zeros(n, dtype=torch.float64, device=_DEV)
    us, roots = [], []
    for _ in range(case["iters"]):
        cost = c - u[nbr]
        near = torch.topk(cost, 3, dim=1, largest=False, sorted=True).values
        lo, hi, s = near[:, 0] - 40 * tau, near[:, 2] + 40 * tau, (near[:, 1] + near[:, 2]) / 2
        going = torch.ones(n, dtype=torch.bool, device=_DEV)
        for _ in range(60):
            g, scale, slope = _logit((s[:, None] - cost) / tau)
            hi = torch.where(going & (g > 0), s, hi)
            lo = torch.where(going & (g <= 0), s, lo)
            new = torch.where(slope > 0, s - g * tau / slope, (lo + hi) / 2)
            small = 4e-16 * (1 + s.abs())
            going = going & (g.abs() > 1e-14 * scale) & ((new - s).abs() > small)
            new = torch.where((new > lo) & (new < hi), new, (lo + hi) / 2)
            going = going & (new != s) & (hi - lo > small)
            s = torch.where(going, new, s)
            if not bool(going.any()):
                break
        us.append(u)
        roots.append(s)
        u = (1 - omega) * u + omega * s
    inst = torch.repeat_interleave(torch.arange(len(offs) - 1, device=_DEV), torch.from_numpy(np.diff(offs)).to(_DEV))
    L = torch.zeros(len(offs) - 1, dtype=torch.float64, device=_DEV)
    L.index_add_(0, inst, 2 * u)
    z = (u[a] + u[b] - ce) / tau
    L.index_add_(0, inst[a], -tau * (z.clamp(min=0.0) + torch.log1p(torch.exp(-z.abs()))))
    out = {"L": L.cpu().numpy()}
    if not case["grad"]:
        return out
    z = (u[:, None] + u[nbr] - c) / tau
    lam = -_logit(z)[0]
    gc = 0.5 * torch.sigmoid(z)
    for u, s in zip(reversed(us), reversed(roots)):
        e = torch.exp(-((s[:, None] + u[nbr] - c) / tau).abs())
        p = e / (1 + e) ** 2 / tau
        total = p.sum(1)
        mu = torch.where(total > 0, omega * lam / total, torch.zeros_like(lam))
        q = mu[:, None] * p
        gc = gc + q
        lam = ((1 - omega) * lam).index_add(0, nbr.reshape(-1), -q.reshape(-1))
    for name, t in (("gx", fx.double()), ("gy", fy.double())):
        slope = torch.where(c > 0, gc * (t[:, None] - t[nbr]) / c, torch.zeros_like(c))
        out[name] = slope.sum(1).index_add(0, nbr.reshape(-1), -slope.reshape(-1)).cpu().numpy()
    return out


def exact(case, seed):
    offs, x, y = _inputs(case, seed)
    n = int(offs[-1])
    if case["kind"] == "smooth":
        return _exact_smooth(case, offs, x, y) if n <= 40000 and len(offs) <= 200 else None
    if case["kind"] == "knn":
        px, py = (torch.from_numpy(q).to(_DEV) for q in (x, y))
        a, b = _union_pairs(px, py, case["top_k"], _dist64)
        d = torch.sort(_dist64(px[a], py[a], px[b], py[b])).values.cpu().numpy()
        Do = np.zeros(case["n"] * case["top_k"])
        Do[:len(d)] = d
        return {"Do": Do, "D": Do / d[0]}
    # the lattice's ties leave the candidate graph to the tie order
    if n > 20000 or len(offs) > 200 or case.get("shape") == "lattice":
        return None
    lp = _exact_lp(case, offs, x, y)
    if lp is None:
        return None
    return {"lp": lp if case["kind"] == "batch" else float(lp[0])}
