"""Performance cases of the power-diagram library: what a program that uses it calls.

`listed()` names the cases, `draw(rng)` gives more of the same ranges,
`prepare(case, seed)` makes a program's inputs and its diagram, `run(state)` is
one pass through the public entry points, `exact(case, seed)` computes the same
outputs by plain torch arithmetic in 64 bits where that is quick enough, and
`work(case)` counts what a pass cannot do without.

Fields of a case
  kind       "eval": masses, centroids and the CSR weight Hessian
             "solve": Newton on the weights, masses at the solved weights
             "derpos": derivatives of masses and centroids with respect to
             positions and weights
  api        "device": the C ABI on device buffers (a program that keeps its
             Diracs on the GPU); "numpy": the Python classes on host arrays
  update     what is new since the last pass: "diracs" (positions and weights)
             or "weights"
  dim, n     dimension, number of Diracs
  points     "uniform"; "clusters": 20 Gaussian clusters mirrored at the box;
             "mix": half uniform, half in clusters clamped to the box;
             "lattice": 70% uniform, 30% on a jittered lattice
  weights    "zero"; "random": uniform in [-1e-6, 1e-6]; "disc": (0.5 / sqrt n)^2
  domain     "box": the unit box, density 1; "poly": the unit cube with density
             1 + 0.3 xyz, normalised; "image": a res x res piecewise-constant
             image of total mass 0.8 with cells clipped by their discs
  precision  "fp64" or "mixed" (FP32 clipping, FP64 re-clip and sums)
  tol        relative mass tolerance of a solve
"""
import ctypes
import math

import numpy as np
import torch

from sdot_b200 import PowerDiagram, _lib
from sdot_b200.optimal_transport import OptimalTransport

BOX = {"domain": "box", "precision": "fp64"}


def listed():
    return [
        # the smallest call: a few hundred cells from a script on numpy arrays
        # (a serving request starts at 1,000 Diracs); latency and launches count
        {"name": "eval2d_numpy_1k", "kind": "eval", "api": "numpy", "update": "diracs", "dim": 2, "n": 1000,
         "points": "uniform", "weights": "zero", **BOX},
        # the plain 2D problem: 10,000 uniform Diracs, one evaluation
        {"name": "eval2d_uniform_10k", "kind": "eval", "api": "device", "update": "diracs", "dim": 2, "n": 10000,
         "points": "uniform", "weights": "zero", **BOX},
        # the caller has its own outer loop on the weights: an odd-sized
        # diagram of which only the weights change from call to call
        {"name": "eval2d_reweight_147k", "kind": "eval", "api": "device", "update": "weights", "dim": 2, "n": 147003,
         "points": "mix", "weights": "random", **BOX},
        # the diagram at scale: the benchmark's workload
        {"name": "eval2d_mix_1M", "kind": "eval", "api": "device", "update": "diracs", "dim": 2, "n": 1000000,
         "points": "mix", "weights": "random", **BOX},
        # the same workload, smaller, on the mixed-precision path
        {"name": "eval2d_mixed_300k", "kind": "eval", "api": "device", "update": "diracs", "dim": 2, "n": 300000,
         "points": "mix", "weights": "random", "domain": "box", "precision": "mixed"},
        # partial transport: an image density, every cell clipped by its disc
        {"name": "eval2d_image_disc_500k", "kind": "eval", "api": "device", "update": "diracs", "dim": 2,
         "n": 500000, "points": "uniform", "weights": "disc", "domain": "image", "precision": "fp64", "res": 512},
        # the 3D workload with its smooth density
        {"name": "eval3d_lattice_200k", "kind": "eval", "api": "device", "update": "diracs", "dim": 3, "n": 200000,
         "points": "lattice", "weights": "zero", "domain": "poly", "precision": "fp64"},
        # a 3D serving request of clustered Diracs: cells on the clusters' rims
        # have hundreds of faces
        {"name": "eval3d_clusters_20k", "kind": "eval", "api": "device", "update": "diracs", "dim": 3, "n": 20011,
         "points": "clusters", "weights": "zero", **BOX},
        # a whole solve, as the example script makes it: 10,000 uniform Diracs to 1e-10
        {"name": "solve2d_uniform_10k", "kind": "solve", "api": "numpy", "update": "weights", "dim": 2, "n": 10000,
         "points": "uniform", "weights": "zero", "tol": 1e-10, **BOX},
        # a larger solve of a serving stream: clustered Diracs, tolerance 1e-8
        {"name": "solve2d_clusters_60k", "kind": "solve", "api": "device", "update": "weights", "dim": 2, "n": 60013,
         "points": "clusters", "weights": "zero", "tol": 1e-8, **BOX},
        # a 3D solve of a serving stream
        {"name": "solve3d_uniform_20k", "kind": "solve", "api": "device", "update": "weights", "dim": 3, "n": 20000,
         "points": "uniform", "weights": "zero", "tol": 1e-8, **BOX},
        # position derivatives: a program that moves its Diracs by gradients
        {"name": "derpos2d_100k", "kind": "derpos", "api": "device", "update": "diracs", "dim": 2, "n": 100001,
         "points": "uniform", "weights": "zero", **BOX},
    ]


def _size(rng, lo, hi):
    """A size in [lo, hi], spread over the logarithm (odd ones among them)."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["eval2d"] * 5 + ["image"] * 2 + ["eval3d"] * 3 + ["solve2d"] * 2 + ["solve3d", "derpos"])
    c = {"kind": "eval", "api": "device", "update": "diracs", "dim": 2, "points": "uniform", "weights": "zero", **BOX}
    if what == "eval2d":
        c["n"] = _size(rng, 1000, 1000000)
        c["api"] = "numpy" if c["n"] < 20000 and rng.random() < 0.3 else "device"
        c["update"] = rng.choice(["diracs", "diracs", "weights"])
        c["points"] = rng.choice(["uniform", "clusters", "mix"])
        c["weights"] = rng.choice(["zero", "random"])
        if c["n"] <= 300000 and rng.random() < 0.2:
            c["precision"] = "mixed"
    elif what == "image":
        c.update(n=_size(rng, 2000, 500000), weights="disc", domain="image", res=_size(rng, 64, 512))
    elif what == "eval3d":
        c.update(dim=3, points=rng.choice(["uniform", "lattice", "clusters"]))
        c["n"] = _size(rng, 1000, 20000 if c["points"] == "clusters" else 200000)
        c["domain"] = rng.choice(["box", "poly"])
        c["update"] = rng.choice(["diracs", "weights"])
    elif what == "solve2d":
        c.update(kind="solve", update="weights", points=rng.choice(["uniform", "clusters"]), tol=1e-8)
        c["n"] = _size(rng, 1000, 60000)
    elif what == "solve3d":
        c.update(kind="solve", update="weights", dim=3, tol=1e-8, n=_size(rng, 1000, 20000))
    else:
        c.update(kind="derpos", n=_size(rng, 1000, 100000))
    return c


# ------------------------------------------------------------------ inputs
def _inputs(case, seed):
    """positions (n, dim) and weights (n) as host arrays, from the seed alone."""
    rng = np.random.Generator(np.random.PCG64(seed))
    n, dim = case["n"], case["dim"]

    def clusters(m):
        centres = rng.random((20, dim))
        return centres[np.arange(m) % 20] + 0.02 * rng.standard_normal((m, dim))

    if case["points"] == "uniform":
        p = rng.random((n, dim))
    elif case["points"] == "clusters":
        p = np.abs(clusters(n))
        p = np.where(p > 1.0, 2.0 - p, p)
    elif case["points"] == "mix":
        p = np.concatenate([rng.random((n // 2, dim)), np.clip(clusters(n - n // 2), 0.0, 1.0)])
    else:  # lattice
        nu = int(round(0.7 * n))
        m = int(math.ceil((n - nu) ** (1.0 / 3.0)))
        g = (np.arange(m) + 0.5) / m
        lat = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[:n - nu]
        p = np.concatenate([rng.random((nu, dim)), lat + rng.uniform(-0.1 / m, 0.1 / m, lat.shape)])
    if case["weights"] == "zero":
        w = np.zeros(n)
    elif case["weights"] == "random":
        w = rng.uniform(-1e-6, 1e-6, n)
    else:
        w = np.full(n, (0.5 / math.sqrt(n)) ** 2)
    return np.ascontiguousarray(p), w


def _image(res):
    x = (np.arange(res) + 0.5) / res
    xx, yy = np.meshgrid(x, x)
    img = 1 + 0.5 * np.sin(6 * np.pi * xx) * np.cos(4 * np.pi * yy)
    return np.ascontiguousarray(img * (0.8 / img.mean()))


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr() if isinstance(t, torch.Tensor) else t.ctypes.data)


class _Diagram:
    """A context of the C ABI and the device buffers a program keeps for it."""

    def __init__(self, case, p, w):
        self.lib = _lib.load()
        self.n, self.dim = p.shape
        prec = _lib.SDOT_MIXED if case["precision"] == "mixed" else _lib.SDOT_FP64
        opt = _lib.SdotOptions(11, None, -1)
        self.ctx = self.lib.sdot_create(self.dim, prec, ctypes.byref(opt))
        if not self.ctx:
            raise RuntimeError("sdot_create failed")
        self.p = torch.from_numpy(p).cuda()
        self.w = torch.from_numpy(w).cuda()
        if case["domain"] == "image":
            img, sizes = _image(case["res"]), np.array([case["res"]] * 2, dtype=np.int64)
            lo, hi = np.zeros(2), np.ones(2)
            self.check(self.lib.sdot_set_image_density(self.ctx, _ptr(lo), _ptr(hi), _ptr(img), _ptr(sizes), 1))
            self.check(self.lib.sdot_set_ball_cut(self.ctx, 1))
        else:
            lo, hi = np.zeros(self.dim), np.ones(self.dim)
            self.check(self.lib.sdot_add_box_shape(self.ctx, _ptr(lo), _ptr(hi), 1.0))
        if case["domain"] == "poly":
            c = np.array([1.0, 0, 0, 0, 0, 0, 0, 0.3]) / (1.0 + 0.3 / 8)
            self.check(self.lib.sdot_set_polynomial_density(self.ctx, _ptr(c), 8))

    def __del__(self):
        if getattr(self, "ctx", None):
            self.lib.sdot_destroy(self.ctx)
            self.ctx = None

    def check(self, st):
        if st != _lib.SDOT_OK:
            raise RuntimeError("status %d: %s" % (st, self.lib.sdot_last_error(self.ctx).decode()))

    def set_diracs(self):
        self.check(self.lib.sdot_set_diracs(self.ctx, _ptr(self.p), _ptr(self.w), self.n, _lib.SDOT_DEVICE))

    def set_weights(self):
        self.check(self.lib.sdot_set_weights(self.ctx, _ptr(self.w), _lib.SDOT_DEVICE))


def _capacity(case):
    return case["n"] * (63 if case["kind"] == "derpos" else 24 if case["dim"] == 3 else 7) + 64


def prepare(case, seed):
    p, w = _inputs(case, seed)
    state = {"case": case, "p": p, "w": w}
    n, dim = p.shape
    # room for the Hessian's entries (the rest of the buffers stays zero): a
    # planar diagram has fewer than 7 per row, a 3D one about 16; a
    # position-derivative block is 9 entries
    cap = state["cap"] = _capacity(case)
    if case["api"] == "numpy":
        if case["kind"] == "solve":
            state["ot"] = OptimalTransport(p, rel_mass_tol=case["tol"])
            state["w0"] = np.zeros(n)
        else:
            pd = PowerDiagram(p, w, precision=case["precision"])
            pd.add_box_shape(np.zeros(dim), np.ones(dim))
            state.update(pd=pd, columns=np.zeros(cap, dtype=np.int64), values=np.zeros(cap))
        return state
    d = _Diagram(case, p, w)
    state["d"] = d
    f, i = {"dtype": torch.float64, "device": "cuda"}, {"dtype": torch.int64, "device": "cuda"}
    state["masses"] = torch.empty(n, **f)
    if case["kind"] == "solve":
        state["target"] = torch.full((n,), 1.0 / n, **f)
        state["out_w"] = torch.empty(n, **f)
        d.set_diracs()
    elif case["kind"] == "derpos":
        state.update(offsets=torch.empty(3 * n + 1, **i), columns=torch.zeros(cap, **i), values=torch.zeros(cap, **f),
                     v=torch.empty(3 * n, **f))
    else:
        state.update(centroids=torch.empty((n, dim), **f), offsets=torch.empty(n + 1, **i),
                     columns=torch.zeros(cap, **i), values=torch.zeros(cap, **f))
        if case["update"] == "weights":
            d.set_diracs()
    torch.cuda.synchronize()
    return state


# -------------------------------------------------------------------- pass
def run(state):
    case = state["case"]
    if case["api"] == "numpy":
        if case["kind"] == "solve":
            ot = state["ot"]
            ot.adjust_weights(initial_weights=state["w0"])
            return {"weights": ot.get_weights(), "masses": ot.get_integrals()}
        pd = state["pd"]
        if case["update"] == "weights":
            pd.set_weights(state["w"])
        else:
            pd.set_positions_and_weights(state["p"], state["w"])
        c = pd.centroids()
        off, col, val, m = pd.der_integrals_wrt_weights()
        state["columns"][:len(col)] = col
        state["values"][:len(val)] = val
        return {"masses": m, "centroids": c, "offsets": off, "columns": state["columns"], "values": state["values"]}
    d = state["d"]
    lib, ctx, dev = d.lib, d.ctx, _lib.SDOT_DEVICE
    if case["kind"] == "solve":
        d.set_weights()
        opt = _lib.SdotNewtonOptions(150, case["tol"], 20000, 1e-12, 1, 0, 0, 0)
        d.check(lib.sdot_solve(ctx, _ptr(state["target"]), dev, ctypes.byref(opt), None))
        d.check(lib.sdot_get_weights(ctx, _ptr(state["out_w"]), dev))
        d.check(lib.sdot_get_integrals(ctx, _ptr(state["masses"]), dev))
        return {"weights": state["out_w"], "masses": state["masses"]}
    if case["update"] == "weights":
        d.set_weights()
    else:
        d.set_diracs()
    nnz = ctypes.c_int64(state["cap"])
    if case["kind"] == "derpos":
        d.check(lib.sdot_get_der_centroids_and_integrals_wrt_weight_and_positions(
            ctx, _ptr(state["offsets"]), _ptr(state["columns"]), _ptr(state["values"]), _ptr(state["v"]),
            ctypes.byref(nnz), dev))
        return {k: state[k] for k in ("offsets", "columns", "values", "v")}
    d.check(lib.sdot_get_centroids(ctx, _ptr(state["centroids"]), None, dev))
    d.check(lib.sdot_get_der_integrals_wrt_weights(ctx, _ptr(state["offsets"]), _ptr(state["columns"]),
                                                   _ptr(state["values"]), _ptr(state["masses"]), ctypes.byref(nnz), 0,
                                                   dev))
    return {k: state[k] for k in ("masses", "centroids", "offsets", "columns", "values")}


# ------------------------------------------------------------------- exact
EXACT_MAX = 12000  # Diracs up to which the brute-force diagram takes a few seconds


def _clip(px, py, ids, cnt, ox, oy, nx, ny, cut):
    """The polygons (rows; cnt valid vertices each) cut by the half-planes
    (o - p) . n >= 0; the new edges get the ids `cut`."""
    cap = px.shape[1]
    k = torch.arange(cap, device=px.device)[None, :]
    valid = k < cnt[:, None]
    d = (ox[:, None] - px) * nx[:, None] + (oy[:, None] - py) * ny[:, None]
    rows = ((d < 0) & valid).any(1).nonzero()[:, 0]
    if rows.numel() == 0:
        return
    d, x, y, e, valid, c = d[rows], px[rows], py[rows], ids[rows], valid[rows], cnt[rows]
    nxt = torch.where(k + 1 < c[:, None], k + 1, torch.zeros_like(k)).clamp(max=cap - 1)
    dn, xn, yn = d.gather(1, nxt), x.gather(1, nxt), y.gather(1, nxt)
    ins, insn = d >= 0, dn >= 0
    keep, cross = valid & ins, valid & (ins != insn)
    t = torch.where(cross, d / (d - dn), torch.zeros_like(d))
    # per vertex: itself when inside, then the crossing of its edge; leaving
    # the half-plane, the new vertex starts the cut's edge, entering it, the rest of its own
    flag = torch.stack([keep, cross], 2).reshape(len(rows), -1)
    ex = torch.stack([x, x + t * (xn - x)], 2).reshape(len(rows), -1)
    ey = torch.stack([y, y + t * (yn - y)], 2).reshape(len(rows), -1)
    ei = torch.stack([e, torch.where(ins, cut[rows][:, None].expand_as(e), e)], 2).reshape(len(rows), -1)
    to = torch.where(flag, flag.long().cumsum(1) - 1, torch.full_like(ei, cap))
    if int(flag.sum(1).max()) > cap:
        raise RuntimeError("a cell has more than %d vertices" % cap)
    for dst, src in ((px, ex), (py, ey), (ids, ei)):
        z = torch.zeros((len(rows), cap + 1), dtype=dst.dtype, device=dst.device)
        z.scatter_(1, to.clamp(max=cap), src)
        dst[rows] = z[:, :cap]
    cnt[rows] = flag.sum(1)


def _diagram2d(p, w, dev):
    """Every cell of the power diagram in the unit box as (x, y, edge ids,
    counts), by clipping with Diracs nearest first until none can reach it."""
    n, cap = len(w), 48
    x0, y0 = p[:, 0], p[:, 1]
    px = torch.zeros((n, cap), dtype=torch.float64, device=dev)
    py, ids = torch.zeros_like(px), torch.full((n, cap), -1, dtype=torch.int64, device=dev)
    px[:, 1:3], py[:, 2:4] = 1.0, 1.0
    cnt = torch.full((n,), 4, dtype=torch.int64, device=dev)
    wmax = w.max()
    active = torch.arange(n, device=dev)
    done = 0
    for upto in (48, 400, n - 1):
        upto = min(upto, n - 1)
        if upto <= done:
            break
        order = torch.empty((len(active), upto), dtype=torch.int64, device=dev)
        dist = torch.empty((len(active), upto), dtype=torch.float64, device=dev)
        for a in range(0, len(active), 1024):
            r = active[a:a + 1024]
            d2 = (x0[r][:, None] - x0) ** 2 + (y0[r][:, None] - y0) ** 2
            d2[torch.arange(len(r), device=dev), r] = math.inf
            v, o = d2.topk(upto, 1, largest=False)
            order[a:a + 1024], dist[a:a + 1024] = o, v
        gx, gy, gi, gc = px[active], py[active], ids[active], cnt[active]
        c0x, c0y, c0w = x0[active], y0[active], w[active]
        for k in range(done, upto):
            j = order[:, k]
            nx, ny = x0[j] - c0x, y0[j] - c0y
            t = 0.5 + 0.5 * (c0w - w[j]) / (nx * nx + ny * ny)
            _clip(gx, gy, gi, gc, c0x + t * nx, c0y + t * ny, nx, ny, j)
        px[active], py[active], ids[active], cnt[active] = gx, gy, gi, gc
        # a Dirac at distance D can cut only if (D - R)^2 - wmax < R^2 - w0
        valid = torch.arange(cap, device=dev)[None, :] < gc[:, None]
        r = torch.where(valid, (gx - c0x[:, None]) ** 2 + (gy - c0y[:, None]) ** 2, torch.zeros_like(gx)).max(1)[0].sqrt()
        far = dist[:, -1].sqrt()
        safe = (far >= r) & ((far - r) ** 2 - wmax >= r * r - c0w) | (gc == 0)
        active, done = active[~safe], upto
        if len(active) == 0:
            break
    return px, py, ids, cnt


def exact(case, seed):
    if case["kind"] == "solve":
        # a solved diagram has its target masses
        return {"weights": None, "masses": np.full(case["n"], 1.0 / case["n"])}
    if case["kind"] != "eval" or case["dim"] != 2 or case["domain"] != "box" or case["n"] > EXACT_MAX:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    hp, hw = _inputs(case, seed)
    p, w = torch.from_numpy(hp).to(dev), torch.from_numpy(hw).to(dev)
    px, py, ids, cnt = _diagram2d(p, w, dev)
    n, cap = px.shape
    k = torch.arange(cap, device=dev)[None, :]
    valid = k < cnt[:, None]
    nxt = torch.where(k + 1 < cnt[:, None], k + 1, torch.zeros_like(k))
    # in coordinates about the Dirac, so that the sums do not cancel
    ux, uy = px - p[:, :1], py - p[:, 1:]
    vx, vy = ux.gather(1, nxt), uy.gather(1, nxt)
    zero = torch.zeros_like(ux)
    cr = torch.where(valid, 0.5 * (ux * vy - uy * vx), zero)
    m = cr.sum(1)
    c = torch.stack([(cr * (ux + vx)).sum(1), (cr * (uy + vy)).sum(1)], 1) / 3
    some = m > 0
    c = torch.where(some[:, None], p + c / torch.where(some, m, torch.ones_like(m))[:, None], torch.zeros_like(c))
    row, e = (valid & (ids >= 0)).nonzero(as_tuple=True)
    j = ids[row, e]
    ln = ((vx - ux)[row, e] ** 2 + (vy - uy)[row, e] ** 2).sqrt()
    h = 0.5 * ln / ((p[row] - p[j]) ** 2).sum(1).sqrt()
    diag = torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, row, h)
    every = torch.arange(n, device=dev)
    key = torch.cat([row * n + j, every * n + every])
    val = torch.cat([-h, diag])[key.argsort()]
    rest = torch.zeros(_capacity(case) - len(val), dtype=torch.float64, device=dev)
    return {"masses": m, "centroids": c, "offsets": None, "columns": None, "values": torch.cat([val, rest])}


# -------------------------------------------------------------------- work
# per cell: the counted operations of the walk (cut attempts, eviction tests,
# final vertices; FMA = 2): 2D uniform, 2D clustered mix, 3D
FLOPS = {"uniform": 3.9e3, "clusters": 2.8e3, "mix": 2.8e3, "3d": 27.5e3}


def work(case):
    n, dim = case["n"], case["dim"]
    flops = n * (FLOPS["3d"] if dim == 3 else FLOPS[case["points"]])
    nnz = n * (16 if dim == 3 else 7)
    if case["kind"] == "derpos":
        return {"bytes": 24 * n + 24 * n + 24 * n + 9 * nnz * 16, "flops": flops + 9 * nnz * 30}
    if case["kind"] == "solve":
        # five Newton steps at least: an evaluation each, the matrix read once
        # per linear solve, the weights and masses out
        return {"bytes": 5 * nnz * 12 + n * 8 * (dim + 4), "flops": 5 * (flops + 2 * nnz)}
    b = n * 8 * (dim + 1) + n * 8 * (dim + 2) + nnz * 16
    if case["domain"] == "image":
        b += 8 * case["res"] ** 2
    return {"bytes": b, "flops": flops}
