"""Performance cases of the CVT engine: what its users run, through its public
entry points, from the smallest drop-in call to the largest grid.

Kinds (the `kind` of a case):

  gcvt     gCVT as the reference's caller uses it: host grids in, host label
           grid out, the energy stop rule, one or more resolution levels
  lloyd    a context's step with inputs in device memory: load, a fixed number
           of Lloyd iterations, the final labels, the run's energy
  charts   the same step over many charts of uneven sizes as one batch
  learned  the step with learned jumps (the shipped network)
  label    one exact labelling of a site grid
  jfa      one jump-flooding labelling of loaded sites
  raster   the density grid of a parameterised mesh
  delaunay the Delaunay triangulation of converged sites
  surface  the stages after the Lloyd loop: the CDT's input points, the
           constrained Delaunay triangulation with the mesh boundary, the lift

Densities are 1 + a sum of Gaussians inside the disk of radius 0.48, sites are
distinct pixels uniform in the disk (the benchmark configurations' family);
everything is made from the seed alone.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "surface-remesher_gb300")
if os.path.join(_PKG, "python") not in sys.path:
    sys.path.insert(0, os.path.join(_PKG, "python"))

import gcvt_gb300 as G  # noqa: E402

MARKER = -32768
RADIUS = 0.48


def listed():
    return [
        # the smallest drop-in call: one small chart through gCVT until its
        # own stop rule ends it; launches and host latency
        dict(name="gcvt_256", kind="gcvt", n=256, sites=300, depth=1, max_iter=1000),
        # a coarse-to-fine drop-in call: three levels, 512 to 2048
        dict(name="gcvt_2048_depth3", kind="gcvt", n=2048, sites=16384, depth=3, max_iter=1000),
        # one ordinary chart, few sites (the benchmark's smallest configuration)
        dict(name="lloyd_1024", kind="lloyd", n=1024, sites=4096, gaussians=8, a_max=4.0,
             s_lo=0.02, s_hi=0.15, iters=50),
        # the benchmark's default configuration
        dict(name="lloyd_4096", kind="lloyd", n=4096, sites=262144, gaussians=32, a_max=8.0,
             s_lo=0.005, s_hi=0.1, iters=100),
        # the largest grid the engine takes
        dict(name="lloyd_8192", kind="lloyd", n=8192, sites=1048576, gaussians=64, a_max=8.0,
             s_lo=0.005, s_hi=0.1, iters=100),
        # a whole atlas: 64 charts of uneven sides in one batch
        dict(name="charts_64", kind="charts", charts=64, max_side=2048, px_per_site=64, iters=100),
        # one chart with learned jumps (the size the shipped network pays at)
        dict(name="learned_1024", kind="learned", n=1024, sites=4096, iters=50, jump_every=4),
        # one labelling of given sites, a side that is no power of two
        dict(name="label_3328", kind="label", n=3328, sites=130000),
        # approximate labels of the default configuration's sites
        dict(name="jfa_4096", kind="jfa", n=4096, sites=262144),
        # the density of a 256 x 256-vertex disk mesh (93,000 triangles)
        dict(name="raster_2048", kind="raster", n=2048, nv=256),
        # triangulating the default configuration's sites after iterations
        dict(name="delaunay_4096", kind="delaunay", n=4096, sites=262144, warm=40),
        # from converged sites to the remeshed surface of that mesh
        dict(name="surface_2048", kind="surface", n=2048, nv=256, px_per_site=48),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["gcvt", "lloyd", "lloyd", "charts", "learned", "label", "jfa", "raster",
                       "delaunay", "surface"])
    side = lambda lo, hi: 256 * max(1, round(_log(rng, lo, hi) / 256))  # noqa: E731
    disk = lambda n, lo, hi: int(math.pi * (RADIUS * n) ** 2 / _log(rng, lo, hi))  # noqa: E731
    if kind == "gcvt":
        n = rng.choice([256, 512, 1024, 2048])
        depth = rng.randint(1, {256: 1, 512: 2, 1024: 3, 2048: 3}[n])
        return dict(kind=kind, n=n, sites=disk(n >> (depth - 1), 40, 200), depth=depth,
                    max_iter=1000)
    if kind == "lloyd":
        n = side(256, 8192)
        return dict(kind=kind, n=n, sites=disk(n, 44, 250), gaussians=rng.randint(4, 64),
                    a_max=round(rng.uniform(2, 8), 2), s_lo=0.01, s_hi=0.12,
                    iters=rng.randint(20, 100))
    if kind == "charts":
        return dict(kind=kind, charts=rng.randint(4, 56), max_side=rng.choice([512, 1024, 2048]),
                    px_per_site=round(_log(rng, 40, 120)), iters=rng.randint(30, 100))
    if kind == "learned":
        n = side(512, 2048)
        return dict(kind=kind, n=n, sites=disk(n, 45, 200), iters=rng.randint(20, 60),
                    jump_every=rng.randint(3, 6))
    if kind == "label":
        n = side(256, 8192)
        return dict(kind=kind, n=n, sites=disk(n, 30, 400))
    if kind == "jfa":
        n = side(256, 8192)
        return dict(kind=kind, n=n, sites=disk(n, 30, 400))
    if kind == "raster":
        return dict(kind=kind, n=16 * round(_log(rng, 256, 4096) / 16),
                    nv=round(_log(rng, 24, 320)))
    if kind == "delaunay":
        n = side(256, 8192)
        return dict(kind=kind, n=n, sites=disk(n, 40, 200), warm=rng.choice([0, 10, 40]))
    n = side(512, 2048)
    return dict(kind=kind, n=n, nv=round(_log(rng, 24, 256)), px_per_site=round(_log(rng, 40, 120)))


# ---- inputs ----------------------------------------------------------------


def _disk(n):
    c = (torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) / n - 0.5
    return c[None, :] ** 2 + c[:, None] ** 2 <= RADIUS * RADIUS


def _density(n, k, a_max, s_lo, s_hi, seed):
    """float32 (n, n): 1 + k seeded Gaussians inside the disk, 0 outside."""
    r = np.random.default_rng([seed, 1])
    a, s = r.uniform(0, a_max, k), r.uniform(s_lo, s_hi, k)
    rad, th = RADIUS * np.sqrt(r.uniform(0, 1, k)), r.uniform(0, 2 * np.pi, k)
    t = lambda v: torch.as_tensor(v, dtype=torch.float64, device="cuda")  # noqa: E731
    mx, my, a, s = t(0.5 + rad * np.cos(th)), t(0.5 + rad * np.sin(th)), t(a), t(s)
    c = (torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) / n
    gx = torch.exp(-((c[:, None] - mx) ** 2) / (2 * s * s))
    gy = torch.exp(-((c[:, None] - my) ** 2) / (2 * s * s))
    rho = 1.0 + (gy * a) @ gx.T
    return torch.where(_disk(n), rho, torch.zeros_like(rho)).float()


def _grid(n, xs, ys):
    """Site grid (n, n, 2) int16 with a site at each (x, y)."""
    g = torch.full((n, n, 2), MARKER, dtype=torch.int16, device="cuda")
    g[ys, xs, 0] = xs.to(torch.int16)
    g[ys, xs, 1] = ys.to(torch.int16)
    return g


def _random_sites(n, m, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed * 7919 + n)
    inside = torch.nonzero(_disk(n).reshape(-1))[:, 0]
    pick = inside[torch.randperm(inside.numel(), generator=gen, device="cuda")[:m]]
    return _grid(n, pick % n, pick // n)


def _mesh(nv, seed):
    """A triangulated unit-disk parameterisation of a height field: uv (V, 2),
    xyz (V, 3), triangles (T, 3), per-vertex density weights (V,)."""
    r = np.random.default_rng([seed, 2])
    h = 1.0 / (nv - 1)
    g = np.arange(nv) * h
    X, Y = np.meshgrid(g, g)
    P = np.stack([X.ravel(), Y.ravel()], 1)
    rr = np.sqrt(((P - 0.5) ** 2).sum(1))
    inside = rr <= RADIUS
    J = r.normal(0.0, 0.3 * h, P.shape)
    # the rim moves less, so that no two boundary edges cross (constraints)
    P = P + np.where((rr > RADIUS - 3 * h)[:, None], 0.24 * h * np.tanh(4 * J / h), J)
    i = np.arange(nv * nv).reshape(nv, nv)
    a, b, c, d = i[:-1, :-1], i[:-1, 1:], i[1:, :-1], i[1:, 1:]
    T = np.concatenate([np.stack([a, b, d], -1).reshape(-1, 3),
                        np.stack([a, d, c], -1).reshape(-1, 3)])
    T = T[inside[T].all(1)]
    used = np.unique(T)
    back = np.full(nv * nv, -1)
    back[used] = np.arange(len(used))
    P, T = P[used], back[T].astype(np.int32)
    f, q, ph = r.uniform(2, 20, 6), r.uniform(2, 20, 6), r.uniform(0, 2 * np.pi, 6)
    z = 0.1 * np.sin(np.outer(P[:, 0], f) + np.outer(P[:, 1], q) + ph).sum(1)
    xyz = np.concatenate([P, z[:, None]], 1)
    e1, e2 = xyz[T[:, 1]] - xyz[T[:, 0]], xyz[T[:, 2]] - xyz[T[:, 0]]
    a3 = 0.5 * np.linalg.norm(np.cross(e1, e2), axis=1)
    a2 = 0.5 * np.abs(e1[:, 0] * e2[:, 1] - e2[:, 0] * e1[:, 1])
    s3, s2 = (np.bincount(T.ravel(), np.repeat(v, 3), len(P)) for v in (a3, a2))
    return P, xyz, T, s3 / s2


def _bary(P, T, t, x, y):
    """Barycentric weights of points (x, y) in triangles t (broadcast)."""
    a, b, c = P[T[t, 0]], P[T[t, 1]], P[T[t, 2]]
    ux, uy, vx, vy = b[..., 0] - a[..., 0], b[..., 1] - a[..., 1], c[..., 0] - a[..., 0], \
        c[..., 1] - a[..., 1]
    px, py = x - a[..., 0], y - a[..., 1]
    det = ux * vy - uy * vx
    w1, w2 = (px * vy - py * vx) / det, (ux * py - uy * px) / det
    return 1 - w1 - w2, w1, w2


def _first_face(P, T, scale, n):
    """Per pixel (x, y) of an n x n grid the first triangle that holds
    (x scale, y scale), len(T) where none does."""
    tri = P[T] / scale
    lo = (tri.amin(1) - 1e-6).ceil().clamp(0, n - 1).long()
    hi = (tri.amax(1) + 1e-6).floor().clamp(0, n - 1).long()
    size = (hi - lo + 1).clamp(min=0)
    count = size[:, 0] * size[:, 1]
    first = torch.full((n * n,), len(T), dtype=torch.int64, device="cuda")
    step = 8192
    for t0 in range(0, len(T), step):
        t = torch.arange(t0, min(t0 + step, len(T)), device="cuda")
        k = torch.repeat_interleave(t, count[t])
        j = torch.arange(len(k), device="cuda") - (count[t].cumsum(0) - count[t])[k - t0]
        x, y = lo[k, 0] + j % size[k, 0], lo[k, 1] + j // size[k, 0]
        inside = torch.stack(_bary(P, T, k, x * scale, y * scale)).amin(0) >= 0
        first.scatter_reduce_(0, (y * n + x)[inside], k[inside], "amin")
    return first


def _raster_inputs(case, seed):
    P, _, T, w = _mesh(case["nv"], seed)
    lo, hi = P.min(0), P.max(0)
    return np.ascontiguousarray(P - lo), w, T, float((hi - lo).max() / (case["n"] - 1))


def _surface_inputs(case, seed):
    """A mesh, its boundary as constraints, and CVT-like sites: a jittered
    triangular lattice over the mesh's pixels, one site per px_per_site."""
    n = case["n"]
    uv, xyz, T, _ = _mesh(case["nv"], seed)
    lo, hi = uv.min(0), uv.max(0)
    scale = float((hi - lo).max() / (n - 1))
    left, lower = float(lo[0]), float(lo[1])
    e = np.concatenate([T[:, [0, 1]], T[:, [1, 2]], T[:, [2, 0]]]).astype(np.int64)
    key = np.sort(e, 1) @ np.array([len(uv), 1])
    _, first, cnt = np.unique(key, return_index=True, return_counts=True)
    be = e[first[cnt == 1]]
    bv = np.unique(be)
    px = ((uv[bv, 0] - left) / scale).astype(np.int64)
    py = ((uv[bv, 1] - lower) / scale).astype(np.int64)
    r = np.random.default_rng([seed, 3])
    h = math.sqrt(case["px_per_site"] * 2 / math.sqrt(3))
    rows = np.arange(0, n / (h * math.sqrt(3) / 2)).astype(np.int64)
    cols = np.arange(0, n / h).astype(np.int64)
    X = (cols[None, :] + 0.5 * (rows[:, None] % 2)) * h
    Y = np.broadcast_to(rows[:, None] * (h * math.sqrt(3) / 2), X.shape)
    q = np.stack([X.ravel(), Y.ravel()], 1)
    q = np.clip(np.rint(q + r.normal(0, 0.12 * h, q.shape)), 0, n - 1).astype(np.int64)
    covered = (_first_face(_cuda(uv - lo), _cuda(T).long(), scale, n) < len(T)).cpu().numpy()
    q = q[covered[q[:, 1] * n + q[:, 0]]]
    fixed = np.unique(py * n + px)
    free = np.setdiff1d(np.unique(q[:, 0] * n + q[:, 1]), (fixed % n) * n + fixed // n)
    return dict(uv=uv, xyz=xyz, T=T, scale=scale, left=left, lower=lower, bv=bv, be=be,
                fixed=fixed, x=free // n, y=free % n)  # free sites in x-major order


def _surface_room(case):
    """Points the surface case's buffers hold: more than any seed's sites and
    boundary vertices."""
    return int(0.9 * case["n"] ** 2 / case["px_per_site"]) + 16 * case["nv"]


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _chart_sides(case):
    sides = [s for s in (256, 512, 1024, 2048) if s <= case["max_side"]]
    return np.random.default_rng(1).choice(sides, case["charts"]).tolist()


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    n = case.get("n")
    if kind == "gcvt":
        # the coarse grid fills the first entries of the site array (depth > 1)
        n0 = n >> (case["depth"] - 1)
        g = np.full((n, n, 2), MARKER, np.int16)
        g.reshape(-1)[:2 * n0 * n0] = _random_sites(n0, case["sites"], seed).cpu().numpy().ravel()
        s.update(sites=g, density=_density(n, 8, 4.0, 0.02, 0.15, seed).cpu().numpy(),
                 mask=np.zeros((n, n), np.uint8), out=np.empty_like(g))
    elif kind in ("lloyd", "learned"):
        k = (case["gaussians"], case["a_max"], case["s_lo"], case["s_hi"]) if kind == "lloyd" \
            else (8, 4.0, 0.02, 0.15)
        s.update(ctx=G.Context(n), sites=_random_sites(n, case["sites"], seed),
                 density=_density(n, *k, seed),
                 mask=torch.zeros((n, n), dtype=torch.uint8, device="cuda"),
                 out=torch.empty((n, n, 2), dtype=torch.int16, device="cuda"))
        if kind == "learned":
            s["ctx"].learning(True)
            s["ctx"].set_mlp(np.load(os.path.join(_PKG, "data", "step_mlp.npy")))
    elif kind == "charts":
        sides = _chart_sides(case)
        out = torch.empty(sum(2 * m * m for m in sides), dtype=torch.int16, device="cuda")
        at, charts = 0, []
        for i, m in enumerate(sides):
            charts.append(dict(
                ctx=G.Context(m), density=_density(m, 8, 4.0, 0.02, 0.15, seed * 64 + i),
                sites=_random_sites(m, int(math.pi * (RADIUS * m) ** 2 / case["px_per_site"]),
                                    seed * 64 + i),
                mask=torch.zeros((m, m), dtype=torch.uint8, device="cuda"),
                out=out[at:at + 2 * m * m].view(m, m, 2)))
            at += 2 * m * m
        s.update(charts=charts, out=out, batch=G.Batch([c["ctx"] for c in charts]))
    elif kind == "label":
        s["sites"] = _random_sites(n, case["sites"], seed)
    elif kind in ("jfa", "delaunay"):
        s["ctx"] = G.Context(n)
        sites, rho = _random_sites(n, case["sites"], seed), _density(n, 16, 8.0, 0.01, 0.12, seed)
        torch.cuda.synchronize()  # the context works on a stream of its own
        s["ctx"].load(sites, rho)
        if case.get("warm"):
            s["ctx"].iterate(case["warm"])
        if kind == "jfa":
            s["out"] = torch.empty((n, n, 2), dtype=torch.int16, device="cuda")
        else:
            s["tri"] = torch.zeros((2 * case["sites"], 3), dtype=torch.int32, device="cuda")
    elif kind == "raster":
        P, w, T, scale = _raster_inputs(case, seed)
        s.update(P=_cuda(P), w=_cuda(w), T=_cuda(T), scale=scale,
                 out=torch.empty((n, n), dtype=torch.float32, device="cuda"))
    elif kind == "surface":
        m = _surface_inputs(case, seed)
        fx, fy = _cuda(m["fixed"] % n), _cuda(m["fixed"] // n)
        mask = torch.zeros((n, n), dtype=torch.uint8, device="cuda")
        mask[fy, fx] = 1
        ctx = G.Context(n)
        sites = _grid(n, torch.cat([_cuda(m["x"]), fx]), torch.cat([_cuda(m["y"]), fy]))
        rho = torch.ones((n, n), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        ctx.load(sites, rho, mask)
        free, con = len(m["x"]), len(m["bv"])
        pos = np.full(len(m["uv"]), -1)
        pos[m["bv"]] = free + np.arange(con)
        room = _surface_room(case)
        cap = 2 * room + 16
        d = dict(dtype=torch.float64, device="cuda")
        s.update(ctx=ctx, scale=m["scale"], left=m["left"], lower=m["lower"], con=con, cap=cap,
                 uv=_cuda(m["uv"]), xyz=_cuda(m["xyz"]), T=_cuda(m["T"]),
                 cpts=_cuda(m["uv"][m["bv"]]), fixed=_cuda(m["bv"].astype(np.int32)),
                 segs=_cuda(pos[m["be"]].astype(np.int32)),
                 points=torch.zeros((room, 2), **d), lifted=torch.zeros((room, 3), **d),
                 tri=torch.zeros((cap, 3), dtype=torch.int32, device="cuda"),
                 face=torch.zeros(room, dtype=torch.int32, device="cuda"),
                 keep=torch.zeros(cap, dtype=torch.uint8, device="cuda"))
    else:
        raise ValueError(kind)
    return s


# ---- one pass --------------------------------------------------------------


def _ok(code, call):
    if code:
        raise G.GcvtError(code, call)


def run(s):
    case = s["case"]
    kind, n = case["kind"], case.get("n")
    lib, dev = G.load_library(), G.MEM_DEVICE
    if kind == "gcvt":
        np.copyto(s["out"], s["sites"])  # gCVT works in place
        return G.gcvt(s["out"], s["density"], s["mask"], case["depth"], case["max_iter"])
    if kind == "lloyd":
        c = s["ctx"]
        c.load(s["sites"], s["density"], s["mask"])
        c.iterate(case["iters"])
        c.label(s["out"])
        return {"labels": s["out"], "energy": c.info()["energy"]}
    if kind == "learned":
        c = s["ctx"]
        c.load(s["sites"], s["density"], s["mask"])
        tried, kept = c.iterate_learned(case["iters"], case["jump_every"])
        c.label(s["out"])
        return {"labels": s["out"], "energy": c.info()["energy"], "tried": tried, "kept": kept}
    if kind == "charts":
        for c in s["charts"]:
            c["ctx"].load(c["sites"], c["density"], c["mask"])
        s["batch"].iterate(case["iters"])
        for c in s["charts"]:
            c["ctx"].label(c["out"])
        return {"labels": s["out"],
                "energy": np.array([c["ctx"].info()["energy"] for c in s["charts"]])}
    if kind == "label":
        return G.label_grid(s["sites"])
    if kind == "jfa":
        _ok(lib.gcvt_ctx_jfa_label(s["ctx"].h, s["out"].data_ptr(), None, dev), kind)
        return s["out"]
    cnt = ctypes.c_int(0)
    if kind == "delaunay":
        _ok(lib.gcvt_ctx_delaunay(s["ctx"].h, s["tri"].data_ptr(), len(s["tri"]),
                                  ctypes.byref(cnt), dev), kind)
        return {"triangles": s["tri"], "count": cnt.value}
    if kind == "raster":
        _ok(lib.gcvt_rasterize(s["P"].data_ptr(), s["w"].data_ptr(), len(s["w"]),
                               s["T"].data_ptr(), len(s["T"]), s["out"].data_ptr(), s["scale"],
                               n, dev), kind)
        return s["out"]
    h, con, frame = s["ctx"].h, s["con"], (s["scale"], s["left"], s["lower"])
    _ok(lib.gcvt_ctx_extract_points(h, *frame, s["points"].data_ptr(), len(s["points"]),
                                    ctypes.byref(cnt), dev), "extract")
    free, pts, det = cnt.value, cnt.value + con, ctypes.c_int(0)
    s["points"][free:pts] = s["cpts"]
    _ok(lib.gcvt_ctx_cdt(h, *frame, s["cpts"].data_ptr(), con, s["segs"].data_ptr(),
                         len(s["segs"]), s["tri"].data_ptr(), s["cap"], ctypes.byref(cnt),
                         ctypes.byref(det), dev), "cdt")
    _ok(lib.gcvt_lift(s["uv"].data_ptr(), s["xyz"].data_ptr(), len(s["uv"]), s["T"].data_ptr(),
                      len(s["T"]), s["points"].data_ptr(), pts, con, s["fixed"].data_ptr(),
                      s["tri"].data_ptr(), cnt.value, s["lifted"].data_ptr(),
                      s["face"].data_ptr(), s["keep"].data_ptr(), dev), "lift")
    return {"points": s["points"], "triangles": s["tri"], "count": cnt.value,
            "lifted": s["lifted"], "face": s["face"], "keep": s["keep"]}


def work(case):
    """Inputs read once, outputs written once; operations: per density pixel and
    iteration the four moment sums (8), per pixel and jump-flooding step nine
    distances (5 each), per rasterised pixel one barycentric evaluation (20),
    per triangle about two incircle tests (40 each)."""
    kind, n = case["kind"], case.get("n", 0)
    nn, disk = n * n, math.pi * RADIUS * RADIUS
    if kind == "gcvt":  # about 70 iterations until the stop rule, most of them coarse
        n0 = n >> (case["depth"] - 1)
        return {"bytes": 13 * nn, "flops": 8 * disk * 70 * n0 * n0}
    if kind in ("lloyd", "learned"):
        return {"bytes": 13 * nn, "flops": 8 * disk * nn * case["iters"]}
    if kind == "charts":
        nn = sum(m * m for m in _chart_sides(case))
        return {"bytes": 13 * nn, "flops": 8 * disk * nn * case["iters"]}
    if kind == "label":
        return {"bytes": 8 * nn, "flops": 5 * nn}
    if kind == "jfa":
        return {"bytes": 4 * nn + nn / 8, "flops": 45 * nn * (int(math.log2(n // 2)) + 2)}
    if kind == "delaunay":
        return {"bytes": nn / 8 + 24 * case["sites"], "flops": 160 * case["sites"]}
    verts = math.pi * (RADIUS * case["nv"]) ** 2
    if kind == "raster":
        return {"bytes": 4 * nn + verts * (24 + 24), "flops": 20 * 0.75 * nn}
    m = 0.75 * nn / case["px_per_site"]
    return {"bytes": nn / 4 + verts * (40 + 24) + m * (16 + 24 + 24 + 4 + 2),
            "flops": 160 * m + 3 * 30 * m}


# ---- the same in 64 bits ---------------------------------------------------


def _exact_raster(case, seed):
    n = case["n"]
    P, w, T, scale = _raster_inputs(case, seed)
    P, w, T = _cuda(P), _cuda(w), _cuda(T).long()
    first = _first_face(P, T, scale, n)
    p = torch.nonzero(first < len(T))[:, 0]
    t = first[p]
    w1, w2, w3 = _bary(P, T, t, (p % n) * scale, (p // n) * scale)
    out = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    out[p] = w1 * w[T[t, 0]] + w2 * w[T[t, 1]] + w3 * w[T[t, 2]]
    return out.view(n, n)


def _exact_surface(case, seed):
    m = _surface_inputs(case, seed)
    free = np.stack([m["x"] * m["scale"] + m["left"], m["y"] * m["scale"] + m["lower"]], 1)
    uv, xyz, T, q = _cuda(m["uv"]), _cuda(m["xyz"]), _cuda(m["T"]).long(), _cuda(free)
    every = torch.arange(len(T), device="cuda")
    lifted = []
    for c in q.split(256):
        w = torch.stack(_bary(uv, T, every, c[:, 0, None], c[:, 1, None]))
        # the first face that holds the point (the nearest to, should rounding
        # leave it in none)
        low = w.amin(0)
        t = torch.where(low >= 0, torch.full_like(low, 2.0), low).argmax(1)
        w = w[:, torch.arange(len(c), device="cuda"), t]
        lifted.append((w[:, :, None] * xyz[T[t]].transpose(0, 1)).sum(0))
    bv, room = _cuda(m["bv"]), _surface_room(case)
    pad = lambda v: torch.nn.functional.pad(v, (0, 0, 0, room - len(v)))  # noqa: E731
    return {"points": pad(torch.cat([q, uv[bv]])), "triangles": None, "count": None,
            "lifted": pad(torch.cat(lifted + [xyz[bv]])), "face": None, "keep": None}


def exact(case, seed):
    if case["kind"] == "raster":
        return _exact_raster(case, seed)
    if case["kind"] == "surface":
        return _exact_surface(case, seed)
    return None  # labels and triangles are whole numbers; an energy is a whole run's
