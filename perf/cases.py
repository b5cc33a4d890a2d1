"""Performance cases of the restricted power diagram engine.

Each case is one call sequence of a user's program through the library's
public boundary (the C ABI of include/rpd.h with device pointers, or the
Python façade where the data lives on the host):

  solve     new seeds -> set_points, launch, moments and statuses
  reweight  new weights for resident seeds (optimal-transport / Lloyd
            iterations) -> set_weights, launch, moments and statuses
  hessian   a Newton step's solve: moments and the facet-area rows
  field     a new implicit domain and new seeds, both on the device
  knn       the K nearest neighbours alone
  batch     many uneven diagrams in one batched launch
  serve     a burst of requests to the serving loop, host data in and out
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(os.getcwd(), "gpu-restricted-power-diagrams_b200"))
sys.path.insert(1, os.path.join(ROOT, "gpu-restricted-power-diagrams_b200"))

import rpd  # noqa: E402
from rpd import synth  # noqa: E402

SCALE = synth.SCALE
PREC = {"fp64": rpd.PRECISION_FP64, "mixed": rpd.PRECISION_MIXED}


def _solve(name, n, seeds, weights, domain, S, K, P=30, V=40, T=100, prec="fp64"):
    return {"name": name, "kind": "solve", "n": n, "seeds": seeds, "weights": weights, "domain": domain, "S": S,
            "K": K, "P": P, "V": V, "T": T, "prec": prec}


def listed():
    return [
        # the smallest diagram a program calls in a loop: latency, launches
        _solve("solve-1k", 1000, "uniform", False, "cube", 16, 50),
        # an ordinary weighted diagram with an odd seed count in the plain box
        _solve("solve-30k-box", 30011, "uniform", True, "none", 0, 70),
        # 100K uniform seeds restricted to a closed blob
        _solve("solve-100k-blob", 100000, "uniform", False, "blob", 100, 70),
        # the 1M-seed weighted lattice in a blob (the benchmark's default)
        _solve("solve-1m-blob", 1000000, "lattice", True, "blob", 200, 50),
        # blue-noise seeds filling the cube, tight caps, large
        _solve("solve-2m-bluenoise", 2000000, "bluenoise", False, "cube", 128, 20, 25, 30),
        # the FP32-filtered predicate
        _solve("solve-250k-mixed", 250000, "uniform", True, "cube", 96, 70, prec="mixed"),
        # a weight-only re-solve of a resident seed set
        {"name": "reweight-300k", "kind": "reweight", "n": 300000, "seeds": "uniform", "domain": "blob", "S": 128,
         "K": 70, "P": 30, "V": 40, "T": 100},
        # a Newton step: facet areas beside the moments
        {"name": "hessian-60k", "kind": "hessian", "n": 60000, "seeds": "lattice", "domain": "cube", "S": 64, "K": 50,
         "P": 30, "V": 40, "T": 100, "H": 40, "HC": 1},
        # a new domain with every solve
        {"name": "field-50k", "kind": "field", "n": 50000, "seeds": "uniform", "S": 80, "K": 50, "P": 30, "V": 40,
         "T": 100},
        # neighbour lists alone
        {"name": "knn-500k", "kind": "knn", "n": 500000, "seeds": "uniform", "K": 50},
        # 48 diagrams of 1K to 200K seeds, K 20, 50 or 70, each in its own blob
        {"name": "batch-48", "kind": "batch", "count": 48, "nmin": 1000, "nmax": 200000, "gmin": 64, "gmax": 160,
         "P": 30, "V": 40, "T": 100},
        # a burst of mixed requests: 9 new diagrams and 3 re-solves
        {"name": "serve-12", "kind": "serve", "new": 9, "again": 3, "nmin": 10000, "nmax": 300000, "K": 50, "P": 30,
         "V": 40, "T": 100, "slots": 4},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "reweight", "hessian", "field", "knn", "batch", "serve"])
    if kind in ("solve", "reweight"):
        n = _logint(rng, 1000, 1000000)
        # dart throwing fills the cube evenly from about 100K points on
        seeds = rng.choice(["uniform", "lattice", "bluenoise" if n >= 100000 else "lattice"])
        domain = rng.choice(["none", "cube", "blob"])
        # voxels about half a cell wide, as the configurations choose them
        S = 0 if domain == "none" else max(12, min(200, int(round(rng.uniform(1.5, 2.2) * n ** (1.0 / 3.0)))))
        K = rng.choice([20, 33, 50, 70]) if seeds != "uniform" else rng.choice([50, 70, 90])
        P, V = rng.choice([(25, 30), (30, 40), (35, 40), (50, 64)])
        if kind == "solve":
            c = _solve("", n, seeds, rng.random() < 0.6, domain, S, K, P, V, rng.choice([60, 100, 150]),
                       rng.choice(["fp64", "fp64", "fp64", "mixed"]))
            del c["name"]
            return c
        return {"kind": kind, "n": n, "seeds": seeds, "domain": domain, "S": S, "K": K, "P": P, "V": V, "T": 100}
    if kind == "hessian":
        n = _logint(rng, 2000, 200000)
        return {"kind": kind, "n": n, "seeds": rng.choice(["uniform", "lattice"]), "domain": rng.choice(["cube", "blob"]),
                "S": max(12, min(128, int(2 * n ** (1.0 / 3.0)))), "K": rng.choice([50, 70]), "P": 30, "V": 40, "T": 100,
                "H": rng.choice([30, 40]), "HC": rng.choice([1, 4])}
    if kind == "field":
        n = _logint(rng, 2000, 300000)
        return {"kind": kind, "n": n, "seeds": rng.choice(["uniform", "lattice"]),
                "S": max(20, min(160, int(2 * n ** (1.0 / 3.0)))), "K": rng.choice([50, 70]), "P": 30, "V": 40, "T": 100}
    if kind == "knn":
        return {"kind": kind, "n": _logint(rng, 2000, 1000000), "seeds": rng.choice(["uniform", "lattice"]),
                "K": rng.choice([8, 20, 33, 50, 70, 100])}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(4, 32), "nmin": 1000, "nmax": _logint(rng, 5000, 150000), "gmin": 48,
                "gmax": 128, "P": 30, "V": 40, "T": 100}
    return {"kind": "serve", "new": rng.randint(2, 8), "again": rng.randint(0, 2), "nmin": 5000,
            "nmax": _logint(rng, 20000, 250000), "K": rng.choice([50, 70]), "P": 30, "V": 40, "T": 100,
            "slots": rng.choice([2, 4])}


# ------------------------------------------------------------------ inputs


def _seeds(kind, n, seed):
    if kind == "uniform":
        return synth.uniform(n, seed=seed)
    if kind == "lattice":
        m = max(2, int(round(n ** (1.0 / 3.0))))
        return synth.jittered_lattice(m, seed=seed, weights=False)
    return synth.poisson_disk(n, seed=seed)


def _weights(n, seed):
    h = n ** (-1.0 / 3.0)
    w = np.random.default_rng(seed + 77).uniform(0.0, 0.1 * h * h, size=n)
    return (w * SCALE * SCALE).astype(np.float32)


def _input(case, seed):
    x = _seeds(case["seeds"], case["n"], seed)
    if case.get("weights", True) and case["kind"] != "knn":
        x[:, 3] = _weights(len(x), seed)
    return x


def _field(S, seed):
    """An implicit domain: a sphere of radius ~0.4 with a seeded ripple."""
    rng = np.random.default_rng(seed + 5)
    a = rng.uniform(0.02, 0.04)
    k = rng.uniform(8.0, 12.0, 3)
    c = rng.uniform(0.47, 0.53, 3)
    g = np.linspace(0.0, 1.0, S + 1)
    z, y, x = np.meshgrid(g, g, g, indexing="ij")
    r = np.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2)
    f = r - 0.4 + a * (np.sin(k[0] * x) * np.sin(k[1] * y) + np.sin(k[2] * z))
    return np.ascontiguousarray(f, np.float32)


def _set_domain(s, case, seed):
    if case["domain"] == "cube":
        s.set_grid(rpd.Grid.cube(case["S"]))
    elif case["domain"] == "blob":
        s.set_grid_blob(case["S"], 5, seed + 11)


def _params(case, **kw):
    return rpd.Params.default(K=case["K"], P=case["P"], V=case["V"], T=case["T"], **kw)


def _dev(a):
    return torch.from_numpy(a).cuda()


def _results(n):
    return torch.zeros((n, 4), dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")


def _ptr(t):
    return rpd.C.c_void_p(t.data_ptr())


def _sizes(case, count):
    """`count` sizes spread evenly over the logarithm of the case's range, in
    a shuffled order that depends on the case alone."""
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    n = [int(round(math.exp(lo + (hi - lo) * (i + 0.5) / count))) for i in range(count)]
    return [n[i] for i in np.random.default_rng(count).permutation(count)]


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "batch":
        # uneven diagrams as the batched workload has them: uniform and
        # jittered-lattice seeds by turns, weights U[0, 0.1 h^2], a blob each
        ctx = rpd.Context(0)
        rng = np.random.default_rng(case["count"])
        sol, par, st["n"] = [], [], []
        for i, n in enumerate(_sizes(case, case["count"])):
            x = _seeds("lattice" if i % 2 else "uniform", n, seed + 1000 * i)
            x[:, 3] = _weights(len(x), seed + 1000 * i)
            S, K = int(rng.integers(case["gmin"], case["gmax"] + 1)), int((20, 50, 70)[int(rng.integers(3))])
            sol.append(rpd.Solver(ctx).set_points(x).set_grid_blob(S, 5, seed + i))
            par.append(rpd.Params.default(K=K, P=case["P"], V=case["V"], T=case["T"]))
            st["n"].append(len(x))
        st["solvers"], st["batch"] = sol, rpd.Batch(sol, par, ctx)
        st["out"], st["status"] = _results(sum(st["n"]))
        return st
    if kind == "serve":
        rng = np.random.default_rng(seed)
        sizes = _sizes(case, case["new"] + case["again"])
        srv = rpd.Server(0, slots=case["slots"])
        grids = {S: rpd.Grid.blob(S, 5, 2) for S in (48, 64, 96, 128)}
        p = _params(case)

        def diagram(k):
            n = sizes[k]
            x = synth.uniform(n, seed=seed + k)
            x[:, 3] = _weights(n, seed + k)
            S = min(grids, key=lambda s: abs(s - 2 * n ** (1.0 / 3.0)))
            return x, grids[S]

        st["requests"] = [diagram(k) for k in range(case["new"])]
        st["resident"] = []
        for k in range(case["again"]):
            x, g = diagram(case["new"] + k)
            t, sess = srv.solve(x, grid=g, params=p)
            srv.wait(t)
            h2 = len(x) ** (-2.0 / 3.0) * SCALE * SCALE
            w = x[:, 3] + (0.01 * h2 * rng.standard_normal(len(x))).astype(np.float32)
            st["resident"].append((sess, np.maximum(w, 0.0).astype(np.float32)))
        st["server"], st["params"] = srv, p
        return st
    x = _input(case, seed)
    n = len(x)
    s = rpd.Solver(rpd.Context(0))
    st.update(solver=s, n=n, x=_dev(x))
    if kind == "knn":
        s.set_points(x)
        st["ids"] = torch.zeros((n, case["K"]), dtype=torch.int32, device="cuda")
        return st
    st["out"], st["status"] = _results(n)
    if kind == "field":
        st["field"] = _dev(_field(case["S"], seed))
        st["params"] = _params(case)
        return st
    _set_domain(s, case, seed)
    if kind == "hessian":
        H, HC = case["H"], case["HC"]
        st["params"] = _params(case, hessian_h=H, hessian_hc=HC)
        st["vals"] = torch.zeros((n, H, HC), dtype=torch.float64, device="cuda")
        st["ids"] = torch.zeros((n, H), dtype=torch.int32, device="cuda")
        return st
    st["params"] = _params(case, precision=PREC[case.get("prec", "fp64")])
    if kind == "reweight":
        s.set_points(x)
        s.launch(st["params"])  # the solve whose seeds and neighbours stay resident
        st["w"] = _dev(_weights(n, seed + 1000))
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    L = rpd.lib()
    if kind == "serve":
        srv, p = st["server"], st["params"]
        tickets, sessions = [], []
        for x, g in st["requests"]:
            t, sess = srv.solve(x, grid=g, params=p)
            tickets.append(t)
            sessions.append(sess)
        for sess, w in st["resident"]:
            tickets.append(srv.reweight(sess, w, p))
        out = [srv.wait(t)[0] for t in tickets]
        for sess in sessions:
            srv.release(sess)
        return out
    if kind == "batch":
        st["batch"].launch()
        a = 0
        for s, n in zip(st["solvers"], st["n"]):
            s.ctx.check(L.rpd_solver_get_moments(s.h, _ptr(st["out"][a:a + n]), rpd.RPD_DEVICE))
            s.ctx.check(L.rpd_solver_get_status(s.h, _ptr(st["status"][a:a + n]), rpd.RPD_DEVICE))
            a += n
        return st["out"], st["status"]
    s, n = st["solver"], st["n"]
    check = s.ctx.check
    if kind == "knn":
        check(L.rpd_solver_knn(s.h, case["K"], _ptr(st["ids"]), rpd.RPD_DEVICE, None))
        return st["ids"]
    if kind == "reweight":
        check(L.rpd_solver_set_weights(s.h, _ptr(st["w"]), rpd.RPD_DEVICE))
    else:
        if kind == "field":
            check(L.rpd_solver_set_grid_field(s.h, case["S"], _ptr(st["field"]), rpd.RPD_DEVICE))
        check(L.rpd_solver_set_points(s.h, _ptr(st["x"]), n, rpd.RPD_DEVICE))
    s.launch(st["params"])
    check(L.rpd_solver_get_moments(s.h, _ptr(st["out"]), rpd.RPD_DEVICE))
    check(L.rpd_solver_get_status(s.h, _ptr(st["status"]), rpd.RPD_DEVICE))
    if kind == "hessian":
        check(L.rpd_solver_get_hessian(s.h, _ptr(st["vals"]), _ptr(st["ids"]), rpd.RPD_DEVICE))
        return st["out"], st["status"], st["vals"], st["ids"]
    return st["out"], st["status"]


def _cells(case):
    if case["kind"] == "batch":
        lo, hi = case["nmin"], case["nmax"]
        return case["count"] * (hi - lo) / math.log(hi / lo) if hi > lo else case["count"] * lo
    if case["kind"] == "serve":
        lo, hi = case["nmin"], case["nmax"]
        return (case["new"] + case["again"]) * (hi - lo) / math.log(hi / lo)
    return case["n"]


def work(case):
    """Seeds (16 bytes) read and moments and status (36 bytes) written once,
    the domain's corner flags and list offsets read once; per cell the about
    27 vertices of a Voronoi cell made (41 operations) and integrated (60)
    and the about 15 faces' planes tested against them (7)."""
    n = _cells(case)
    if case["kind"] == "knn":
        return {"bytes": n * (16 + 4 * case["K"]), "flops": n * case["K"] * 8.0}
    b = n * (16 + 36)
    if case["kind"] == "hessian":
        b += n * case["H"] * (8 * case["HC"] + 4)
    if case["kind"] == "field":
        b += 4 * (case["S"] + 1) ** 3
    elif case["kind"] in ("solve", "reweight", "hessian"):
        b += 5 * case["S"] ** 3
    return {"bytes": float(b), "flops": n * 27 * (41 + 60 + 15 * 7.0)}


# ------------------------------------------------- the same in 64 bits


def _exact_cells(x, lo, hi, K, want_area):
    """Moments (and per neighbour, nearest first, the facet areas) of the
    power cells of seeds x (n, 4) restricted to the box [lo, hi]^3, from the
    K nearest neighbours' bisectors: every edge of a cell is the line of two
    of its planes, cut by all others; each adds the signed tetrahedron of the
    seed, the foot of the seed on the face's plane, and the edge."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    X = torch.from_numpy(np.asarray(x, np.float64)).to(dev)
    n = len(X)
    P, W = X[:, :3], X[:, 3]
    K = min(K, n - 1)
    out = torch.zeros((n, 4), dtype=torch.float64, device=dev)
    areas = torch.zeros((n, K), dtype=torch.float64, device=dev) if want_area else None
    step = 32
    for a in range(0, n, step):
        b = min(n, a + step)
        s, ws = P[a:b], W[a:b]
        d2 = ((s[:, None, :] - P[None, :, :]) ** 2).sum(-1)
        d2[torch.arange(b - a, device=dev), torch.arange(a, b, device=dev)] = math.inf
        d2, idx = d2.topk(K, largest=False, sorted=True)
        v = P[idx] - s[:, None, :]
        ln = d2.sqrt()
        nb = -v / ln[..., None]
        ob = (d2 + W[idx] - ws[:, None]) / (2.0 * ln)
        eye = torch.eye(3, dtype=torch.float64, device=dev)
        bx = torch.cat([eye, -eye])[None].expand(b - a, 6, 3)
        obx = torch.cat([s - lo, hi - s], 1)
        N = torch.cat([bx, nb], 1)  # inward unit normals: N . p + D >= 0
        D = torch.cat([obx, ob], 1)
        M = N.shape[1]
        # only planes nearer than the cell's reach matter; all are kept
        dirs = torch.cross(N[:, :, None, :].expand(-1, M, M, 3), N[:, None, :, :].expand(-1, M, M, 3), dim=-1)
        dd = (dirs * dirs).sum(-1)
        ok = dd > 1e-18
        ddi = torch.where(ok, 1.0 / dd.clamp_min(1e-300), torch.zeros_like(dd))
        n1, n2 = N[:, :, None, :].expand_as(dirs), N[:, None, :, :].expand_as(dirs)
        p0 = (-D[:, :, None, None] * torch.cross(n2, dirs, dim=-1) - D[:, None, :, None] * torch.cross(dirs, n1, dim=-1))
        p0 = p0 * ddi[..., None]
        val = torch.einsum("bfgc,bhc->bfgh", p0, N) + D[:, None, None, :]
        sl = torch.einsum("bfgc,bhc->bfgh", dirs, N)
        i = torch.arange(M, device=dev)
        skip = (i[:, None, None] == i[None, None, :]) | (i[None, :, None] == i[None, None, :])
        flat = sl.abs() <= 1e-14
        t = -val / torch.where(flat, torch.ones_like(sl), sl)
        inf = torch.full_like(t, math.inf)
        low = torch.where(skip | flat | (sl < 0), -inf, t).amax(-1)
        high = torch.where(skip | flat | (sl > 0), inf, t).amin(-1)
        dead = (flat & ~skip & (val < -1e-12)).any(-1)
        on = ok & ~dead & (low < high) & torch.isfinite(low) & torch.isfinite(high)
        low, high = torch.where(on, low, 0.0), torch.where(on, high, 0.0)
        U = p0 + low[..., None] * dirs
        V = p0 + high[..., None] * dirs
        C = (-D[..., None] * N)[:, :, None, :].expand_as(U)
        det = (C * torch.cross(U, V, dim=-1)).sum(-1) / 6.0
        det = torch.where(on, det, 0.0)
        m = det.sum((1, 2))
        mom = (det[..., None] * (C + U + V) * 0.25).sum((1, 2))
        sgn = torch.sign(m)
        m, mom = m * sgn, mom * sgn[:, None]
        out[a:b, 3] = m
        out[a:b, :3] = mom + m[:, None] * s
        if want_area:
            ar = 0.5 * (torch.cross(U - C, V - C, dim=-1) * n1).sum(-1)
            areas[a:b] = torch.where(on, ar, 0.0).sum(2).abs()[:, 6:]
    return out, areas


def exact(case, seed):
    """Cells in the box or the cube domain (whose restriction is a smaller
    box) for sizes that take seconds; the other domains' surfaces are this
    library's own triangulations, neighbour lists and statuses whole
    numbers."""
    if case["kind"] not in ("solve", "hessian", "reweight") or case["domain"] == "blob" or case["n"] > 60000:
        return None
    x = _input(case, seed)
    if case["kind"] == "reweight":
        x[:, 3] = _weights(len(x), seed + 1000)
    lo = 500.0 / case["S"] if case["domain"] == "cube" else 0.0
    hi = SCALE - lo
    out, areas = _exact_cells(x, lo, hi, 112, case["kind"] == "hessian" and case["HC"] == 1)
    if case["kind"] != "hessian":
        return out, None
    if areas is None:
        return out, None, None, None
    H = case["H"]
    vals = torch.zeros((len(x), H, 1), dtype=torch.float64, device=out.device)
    keep = areas > 0.2
    pos = keep.cumsum(1) - 1
    r, c = torch.nonzero(keep & (pos < H), as_tuple=True)
    vals[r, pos[r, c], 0] = areas[r, c]
    return out, None, vals, None
