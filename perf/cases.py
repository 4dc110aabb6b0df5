"""The work a user of this package has it do, through its public entry points.

Every case is one of five kinds:

* ``reduce``  one filtered complex, its boundary matrix in hand: the MEX-shaped
  call ``ph`` (1-based COO on the host), ``Context.reduce`` (CSC on the host)
  or ``Context.reduce_device`` (CSC in device memory);
* ``points``  a point cloud on the device to its persistence pairs: the Rips
  complex built there, then reduced;
* ``image``   an image on the device to its persistence pairs (lower star);
* ``batch``   many Rips complexes in one segmented call, host or device;
* ``serve``   a stream of requests through ``Server``.

The shapes are the package's own benchmark and test shapes (``complexes``):
Rips complexes of points in a cube, on a noisy circle and on a torus, and
lower-star filtrations of smoothed images.  One ``Context`` and one ``Server``
are kept for the process, as a program that reduces more than one complex
keeps them.
"""
import math

import numpy as np
import torch

from openph_gb300 import api
from openph_gb300 import complexes as cx

_kept = {}


def _context():
    if "context" not in _kept:
        _kept["context"] = api.Context(0)
    return _kept["context"]


def _server():
    if "server" not in _kept:
        _kept["server"] = api.Server(0, budget_bytes=8 << 30)
    return _kept["server"]


def listed():
    return [
        # the smallest call there is in earnest: a dozen points, all latency
        {"name": "rips_12_device", "kind": "reduce", "shape": "cube", "n": 12, "algo": "pms", "via": "device"},
        # the 20,875-column configuration, through the reference's own call
        {"name": "rips_cube_50_ph", "kind": "reduce", "shape": "cube", "n": 50, "algo": "pms", "via": "ph"},
        # an ordinary complex, from host memory to host memory
        {"name": "torus_200k_host", "kind": "reduce", "shape": "torus", "n": 400, "m": 200_000, "algo": "pms",
         "via": "host"},
        # the five-million-column configuration
        {"name": "torus_5m_device", "kind": "reduce", "shape": "torus", "n": 400, "m": 5_000_000, "algo": "pms",
         "via": "device"},
        # the 512 x 512 image configuration
        {"name": "lower_star_512_device", "kind": "reduce", "shape": "image", "h": 512, "w": 512, "algo": "pms",
         "via": "device"},
        # a cloud of points to its pairs, nothing leaving the device
        {"name": "points_torus_1m", "kind": "points", "n": 400, "m": 1_000_000},
        # an image of odd sides to its pairs
        {"name": "image_97x203", "kind": "image", "h": 97, "w": 203},
        # the batched configuration's mix, a quarter of its complexes
        {"name": "batch_1024_device", "kind": "batch", "count": 1024, "lo": 20, "hi": 120, "via": "device"},
        # a small batch from host memory
        {"name": "batch_40_host", "kind": "batch", "count": 40, "lo": 20, "hi": 60, "via": "host"},
        # a burst of mixed requests on the server
        {"name": "serve_24", "kind": "serve", "count": 24, "lo": 1_000, "hi": 500_000},
        # the column-by-column algorithms, which the reference's users compare with pms
        {"name": "twist_image_64_ph", "kind": "reduce", "shape": "image", "h": 64, "w": 64, "algo": "twist",
         "via": "ph"},
        {"name": "standard_cube_24_host", "kind": "reduce", "shape": "cube", "n": 24, "algo": "standard",
         "via": "host"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["reduce", "reduce", "reduce", "points", "image", "batch", "serve", "sequential"])
    if kind == "sequential":
        algo = rng.choice(["twist", "standard", "ph_row", "twist_parallel", "standard_parallel", "ph_row_parallel"])
        via = rng.choice(["ph", "host"])
        if rng.random() < 0.5:
            return {"kind": "reduce", "shape": rng.choice(["cube", "circle"]), "n": rng.randint(12, 30), "algo": algo,
                    "via": via}
        return {"kind": "reduce", "shape": "image", "h": rng.randint(9, 48), "w": rng.randint(9, 48), "algo": algo,
                "via": via}
    if kind == "reduce":
        shape, via = rng.choice(["cube", "circle", "torus", "image"]), rng.choice(["ph", "host", "device", "device"])
        case = {"kind": kind, "shape": shape, "algo": "pms", "via": via}
        if shape == "torus":
            return dict(case, n=rng.randint(250, 400), m=_log_uniform(rng, 50_000, 2_500_000))
        if shape == "image":
            return dict(case, h=_log_uniform(rng, 10, 512), w=_log_uniform(rng, 10, 512))
        return dict(case, n=_log_uniform(rng, 10, 200))
    if kind == "points":
        return {"kind": kind, "n": rng.randint(250, 400), "m": _log_uniform(rng, 50_000, 2_500_000)}
    if kind == "image":
        return {"kind": kind, "h": _log_uniform(rng, 10, 512), "w": _log_uniform(rng, 10, 512)}
    if kind == "batch":
        return {"kind": kind, "count": _log_uniform(rng, 8, 512), "lo": rng.randint(5, 30), "hi": rng.randint(40, 120),
                "via": rng.choice(["host", "device", "device"])}
    return {"kind": kind, "count": rng.randint(6, 24), "lo": _log_uniform(rng, 500, 2_000),
            "hi": _log_uniform(rng, 50_000, 500_000)}


# ------------------------------------------------------------------- inputs
def _torus_points(n, seed):
    return cx.points_torus(n, seed)


def _matrix(case, seed):
    """The boundary matrix of a ``reduce`` case, on the host."""
    shape = case["shape"]
    if shape == "image":
        img = cx.image_smoothed(case["h"], case["w"], seed)
        return cx.lower_star_device(torch.from_numpy(img).cuda(), ctx=_context()).to_host()
    if shape != "torus":
        pts = cx.points_cube(case["n"], seed) if shape == "cube" else cx.points_circle(case["n"], seed)
        return cx.rips_device(torch.from_numpy(pts).cuda(), math.inf, ctx=_context()).to_host()
    # the first case["m"] simplices of the filtration: a complex again, of the
    # same size for every seed
    m, pts = case["m"], _torus_points(case["n"], seed)
    thr = cx.rips_threshold(pts, m + m // 50 + 1000)
    bm = cx.rips_device(torch.from_numpy(pts).cuda(), thr, ctx=_context()).to_host()
    return cx.BoundaryMatrix(bm.colptr[:m + 1], bm.rows[:bm.colptr[m]])


def _room(case):
    """Columns the buffers of a ``points`` case hold."""
    return case["m"] + case["m"] // 10 + 1000


def _request_sizes(case):
    """Target column counts of a stream's requests, spread over their logarithm."""
    k = case["count"]
    return [int(round(case["lo"] * (case["hi"] / case["lo"]) ** (i / max(1, k - 1)))) for i in range(k)]


def _request(i, m, seed):
    """Request i of a stream: the three configurations' shapes in turn."""
    if i % 3 == 0:
        return {"kind": "reduce", "shape": "cube", "n": max(6, int(round((6 * m) ** (1 / 3))))}
    if i % 3 == 1:
        side = max(4, int(round((m / 6) ** 0.5)))
        return {"kind": "reduce", "shape": "image", "h": side, "w": side + 1}
    return {"kind": "reduce", "shape": "torus", "n": 200 if m < 50_000 else 400, "m": m}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "points":
        # buffers with room to spare: the complex's size follows from the points
        pts, room = _torus_points(case["n"], seed), _room(case)
        return {"kind": kind, "ctx": _context(), "points": torch.from_numpy(pts).cuda(),
                "threshold": cx.rips_threshold(pts, case["m"]),
                "colptr": torch.zeros(room + 1, dtype=torch.int64, device="cuda"),
                "rows": torch.zeros(3 * room, dtype=torch.int32, device="cuda"),
                "values": torch.zeros(room, dtype=torch.float64, device="cuda"),
                "low": torch.zeros(room, dtype=torch.int32, device="cuda"),
                "ess": torch.zeros(room, dtype=torch.int32, device="cuda")}
    if kind == "image":
        return {"kind": kind, "ctx": _context(),
                "image": torch.from_numpy(cx.image_smoothed(case["h"], case["w"], seed)).cuda()}
    if kind == "batch":
        # point counts spread evenly over [lo, hi] in a fixed order, half of the
        # complexes in the cube and half on the circle (by the seeds' parity)
        sizes = np.random.default_rng(4).permutation(np.linspace(case["lo"], case["hi"], case["count"]).astype(np.int32))
        seeds = np.arange(case["count"], dtype=np.uint64) + np.uint64(seed) * np.uint64(100_003)
        col_off, colptr, rows = cx.rips_mixed_instances(sizes, seeds)
        state = {"kind": kind, "via": case["via"], "ctx": _context(), "count": case["count"], "m": int(col_off[-1]),
                 "nnz": int(colptr[-1])}
        if case["via"] == "host":
            return dict(state, col_off=col_off, colptr=colptr, rows=rows)
        out = torch.empty(2, max(1, state["m"]), dtype=torch.int32, device="cuda")
        return dict(state, col_off=torch.from_numpy(col_off).cuda(), colptr=torch.from_numpy(colptr).cuda(),
                    rows=torch.from_numpy(rows).cuda(), low=out[0], ess=out[1])
    if kind == "serve":
        mats = [_matrix(_request(i, m, seed), seed * 1000 + i) for i, m in enumerate(_request_sizes(case))]
        return {"kind": kind, "server": _server(), "mats": mats}
    bm = _matrix(case, seed)
    state = {"kind": kind, "via": case["via"], "algo": case["algo"], "ctx": _context(), "m": bm.m}
    if case["via"] == "ph":
        r, c = bm.to_coo1()
        return dict(state, r=r, c=c)
    if case["via"] == "host":
        return dict(state, bm=bm)
    return dict(state, colptr=torch.from_numpy(bm.colptr).cuda(), rows=torch.from_numpy(bm.rows).cuda(),
                low=torch.empty(bm.m, dtype=torch.int32, device="cuda"),
                ess=torch.empty(bm.m, dtype=torch.int32, device="cuda"))


# ---------------------------------------------------------------------- run
def run(state):
    kind, ctx = state["kind"], state.get("ctx")
    if kind == "points":
        out = [state[k] for k in ("colptr", "rows", "values", "low", "ess")]
        p = [x.data_ptr() for x in out]
        n, d = state["points"].shape
        m, _ = ctx.rips_device(state["points"].data_ptr(), n, d, state["threshold"], lambda m, nnz: p[:3])
        ctx.reduce_device(m, p[0], p[1], p[3], p[4])
        return out
    if kind == "image":
        dm = cx.lower_star_device(state["image"], ctx=ctx)
        low = torch.empty(dm.m, dtype=torch.int32, device="cuda")
        ess = torch.empty(dm.m, dtype=torch.int32, device="cuda")
        ctx.reduce_device(dm.m, dm.colptr.data_ptr(), dm.rows.data_ptr(), low.data_ptr(), ess.data_ptr())
        return [dm.colptr, dm.rows, dm.values, low, ess]
    if kind == "batch":
        if state["via"] == "host":
            low, ess, _ = ctx.reduce_batch_packed(state["col_off"], state["colptr"], state["rows"])
            return [low, ess]
        ctx.reduce_batch_device(state["count"], state["col_off"].data_ptr(), state["colptr"].data_ptr(),
                                state["rows"].data_ptr(), state["m"], state["nnz"], state["low"].data_ptr(),
                                state["ess"].data_ptr())
        return [state["low"], state["ess"]]
    if kind == "serve":
        server = state["server"]
        tickets = [server.submit(bm) for bm in state["mats"]]
        return [list(server.wait(t)[:2]) for t in tickets]
    if state["via"] == "ph":
        out = api.ph(state["algo"], state["r"], state["c"], state["m"])
        return [out[0], out[1]]
    if state["via"] == "host":
        low, ess, _ = ctx.reduce(state["bm"], state["algo"])
        return [low, ess]
    ctx.reduce_device(state["m"], state["colptr"].data_ptr(), state["rows"].data_ptr(), state["low"].data_ptr(),
                      state["ess"].data_ptr(), algo=state["algo"])
    return [state["low"], state["ess"]]


# --------------------------------------------------------------------- work
def _size(case):
    """Columns and nonzeros of a ``reduce``, ``points`` or ``image`` case."""
    if "h" in case:
        h, w = case["h"], case["w"]
        d = (h - 1) * (w - 1)
        e = h * (w - 1) + (h - 1) * w + d
        return h * w + e + 2 * d, 2 * e + 6 * d
    if "m" in case:
        return case["m"], 3 * case["m"]
    n = case["n"]
    e, t = n * (n - 1) // 2, n * (n - 1) * (n - 2) // 6
    return n + e + t, 2 * e + 3 * t


def work(case):
    """Bytes of one pass: the matrix read once and low and ess written once (and
    a complex built on the way written once); the additions over Z/2 that a
    reduction needs depend on the data and are not counted."""
    kind = case["kind"]
    if kind == "batch":
        sizes = [_size({"n": int(n)}) for n in np.linspace(case["lo"], case["hi"], case["count"])]
        m, nnz = (sum(s[i] for s in sizes) for i in (0, 1))
        return {"bytes": 16 * m + 4 * nnz, "flops": 0}
    if kind == "serve":
        sizes = [_size(_request(i, m, 0)) for i, m in enumerate(_request_sizes(case))]
        return {"bytes": sum(16 * m + 4 * nnz for m, nnz in sizes), "flops": 0}
    m, nnz = _size(case)
    if kind in ("points", "image"):  # the matrix and its values written, then the pairs
        return {"bytes": 24 * m + 4 * nnz, "flops": 0}
    return {"bytes": (8 * nnz if case["via"] == "ph" else 8 * m + 4 * nnz) + 8 * m, "flops": 0}


# -------------------------------------------------------------------- exact
def _reduced(colptr, rows):
    """Lows (0-based, -1 = none) and essential flags by the textbook reduction,
    columns as Python integers, top dimension first with clearing."""
    m = len(colptr) - 1
    size = np.diff(colptr)
    low, ess, owner = np.full(m, -1, np.int32), np.ones(m, np.int32), {}
    for d in sorted(set(size[size > 0].tolist()), reverse=True):
        for j in np.flatnonzero(size == d).tolist():
            if ess[j] == 0:  # some column's low: it reduces to zero
                continue
            col = 0
            for r in rows[colptr[j]:colptr[j + 1]].tolist():
                col ^= 1 << r
            while col and (col.bit_length() - 1) in owner:
                col ^= owner[col.bit_length() - 1]
            if col:
                i = col.bit_length() - 1
                owner[i] = col
                low[j], ess[i], ess[j] = i, 0, 0
    return low, ess


def _rips_values(pts, thr):
    """The filtration values of a Rips complex, ascending."""
    sq = np.zeros((len(pts), len(pts)))
    for t in range(pts.shape[1]):
        sq = sq + (pts[:, None, t] - pts[None, :, t]) ** 2
    dist = np.sqrt(sq)
    a, b = np.nonzero(np.triu(dist <= thr, 1))
    tri = []
    for i in range(len(pts)):
        near = np.flatnonzero((dist[i] <= thr) & (np.arange(len(pts)) > i))
        p, q = np.triu_indices(len(near), 1)
        v = np.maximum(np.maximum(dist[i, near[p]], dist[i, near[q]]), dist[near[p], near[q]])
        tri.append(v[dist[near[p], near[q]] <= thr])
    return np.sort(np.concatenate([np.zeros(len(pts)), dist[a, b], *tri]))


def _image_values(img):
    """The filtration values of an image's lower-star complex, ascending."""
    f = img.astype(np.float64)
    h, v = np.maximum(f[:, :-1], f[:, 1:]), np.maximum(f[:-1], f[1:])
    diag = np.maximum(f[:-1, :-1], f[1:, 1:])
    up, down = np.maximum(diag, f[:-1, 1:]), np.maximum(diag, f[1:, :-1])
    return np.sort(np.concatenate([x.ravel() for x in (f, h, v, diag, up, down)]))


def exact(case, seed):
    kind = case["kind"]
    if kind == "points":
        pts, values = _torus_points(case["n"], seed), np.zeros(_room(case))
        v = _rips_values(pts, cx.rips_threshold(pts, case["m"]))
        values[:len(v)] = v
        return [None, None, values, None, None]
    if kind == "image":
        return [None, None, _image_values(cx.image_smoothed(case["h"], case["w"], seed)), None, None]
    if kind != "reduce" or _size(case)[0] > 25_000:
        return None
    bm = _matrix(case, seed)
    low, ess = _reduced(bm.colptr, bm.rows)
    if case["algo"] in ("ph_row", "ph_row_parallel"):  # the row forms keep an estimate of their own
        ess = None
    if case["via"] == "ph":
        low = low + 1
    return [low, ess]
