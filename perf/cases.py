"""The work whose speed matters here, as a list of cases over the framework's public API.

A case is a dict of plain values.  `listed()` gives the cases that are followed from one
version to the next, `draw(rng)` further ones of the same ranges, `prepare(case, seed)` what
a program holds before the call, `run(state)` one pass, `work(case)` the bytes and operations
a pass cannot do without, `exact(case, seed)` the same results from plain numpy in 64 bits
where that takes seconds at most.

Kinds of case:
  solve    TerrainGenerator.generate() on a model that stays on the GPU
  grid     the same on a triangulated height-map lattice, page-locked host arrays
  fresh    a model put on the GPU, solved once and dropped (one terrain per program)
  batch    BatchGenerator.generate(): many terrains in one packed solve
  served   a burst of requests of mixed sizes to a TerrainServer
  profile  get_elevations() at a few points, host arrays
  render   interpolate_device() of a square pixel grid, arrays on the GPU
Sizes follow fastlem_gb300/workloads.py and the tests: 10,000 sites (the reference's CPU
example), 1,000,000, 16,000,000, batches of 4,096..262,144 sites, requests from 16,384.
"""
import math

import numpy as np
import torch

from fastlem_gb300 import (ParameterArrays, Site2D, Terrain2D, TerrainGenerator, TerrainModel2D,
                           TerrainModel2DBulider, pinned_empty)
from fastlem_gb300.api import TerrainInterpolator2D
from fastlem_gb300.batch import BatchGenerator, TerrainBatch
from fastlem_gb300.serve import TerrainServer

SLOPE = 3.14 * 0.1            # the slope limit of the reference's example


def listed():
    return [
        # the smallest terrains: an interactive preview after each change of a parameter
        {"name": "solve_1k", "kind": "solve", "n": 1000, "relax": 1, "slope": False,
         "outlets": "border", "iters": 0},
        # the reference's CPU example size, run until nothing changes (the default)
        {"name": "solve_10k", "kind": "solve", "n": 10000, "relax": 1, "slope": False,
         "outlets": "border", "iters": 0},
        # the reference's slope-limited example: outlets from the hull, a limit on every site
        # (with a rough erodibility field such a terrain may swing for ever: bounded)
        {"name": "solve_10k_slope", "kind": "solve", "n": 10007, "relax": 1, "slope": True,
         "outlets": "hull", "iters": 100},
        # an ordinary map, an odd number of sites, run until nothing changes
        {"name": "solve_65k", "kind": "solve", "n": 65537, "relax": 0, "slope": False,
         "outlets": "border", "iters": 0},
        # a larger map with slope limits and a bounded number of iterations
        {"name": "solve_250k_slope", "kind": "solve", "n": 250007, "relax": 0, "slope": True,
         "outlets": "border", "iters": 32},
        # the million-site configuration with a bounded number of iterations
        {"name": "solve_1m", "kind": "solve", "n": 1000000, "relax": 0, "slope": False,
         "outlets": "border", "iters": 64},
        # the largest: 16 million sites of a triangulated height map, eight iterations
        {"name": "grid_16m", "kind": "grid", "w": 4099, "h": 3907, "iters": 8},
        # a program that builds one model, solves it once and ends
        {"name": "fresh_100k", "kind": "fresh", "n": 100003, "iters": 32},
        # a set of independent maps (training data, variations of one world) to convergence
        {"name": "batch_48", "kind": "batch", "terrains": 48, "lo": 4096, "hi": 131072, "iters": 0},
        # a burst of requests of mixed sizes
        {"name": "served_24", "kind": "served", "requests": 24, "lo": 16384, "hi": 262144,
         "iters": 64},
        # elevations along a path: few queries, arrays on the host
        {"name": "profile_1500", "kind": "profile", "n": 10000, "queries": 1500},
        # a rendered picture of a finished terrain, arrays on the GPU
        {"name": "render_2048", "kind": "render", "n": 250000, "px": 2048},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve"] * 6 + ["grid", "fresh", "batch", "batch", "served", "profile", "render"])
    if kind == "solve":
        n = _log(rng, 300, 1000000)
        # to convergence where that is an ordinary wait, else a bounded number of iterations
        slope = rng.random() < 0.3
        iters = 0 if n <= 70000 and not slope and rng.random() < 0.8 else rng.randint(4, 64)
        return {"kind": kind, "n": n, "relax": rng.choice([0, 1]) if n <= 100000 else 0,
                "slope": slope, "outlets": rng.choice(["border", "border", "hull"]),
                "iters": iters}
    if kind == "grid":
        w = _log(rng, 700, 4099)
        return {"kind": kind, "w": w, "h": max(500, int(w * rng.uniform(0.6, 0.95))),
                "iters": rng.randint(2, 8)}
    if kind == "fresh":
        return {"kind": kind, "n": _log(rng, 2000, 400000), "iters": rng.randint(4, 32)}
    if kind == "batch":
        lo = _log(rng, 1024, 8192)
        return {"kind": kind, "terrains": rng.randint(3, 48), "lo": lo,
                "hi": lo * rng.randint(2, 16), "iters": rng.choice([0, rng.randint(8, 64)])}
    if kind == "served":
        lo = _log(rng, 4096, 16384)
        return {"kind": kind, "requests": rng.randint(4, 24), "lo": lo, "hi": lo * rng.randint(2, 16),
                "iters": rng.randint(8, 64)}
    if kind == "profile":
        return {"kind": kind, "n": _log(rng, 1000, 200000), "queries": _log(rng, 1, 20000)}
    return {"kind": kind, "n": _log(rng, 2000, 250000), "px": _log(rng, 64, 2048)}


# ---- inputs ------------------------------------------------------------------------

def _model(n, side, seed, relax=0):
    b = TerrainModel2DBulider.from_random_sites(n, Site2D(0.0, 0.0), Site2D(side, side), seed=seed)
    return (b.relaxate_sites(relax) if relax else b).build()


def _border(m, side):
    w = 0.02 * side
    return (m.xs < w) | (m.xs > side - w) | (m.ys < w) | (m.ys > side - w)


def _lognormal(n, seed):
    return np.exp(np.random.default_rng(seed).normal(0.0, 0.5, n))


def _solve_inputs(c, seed):
    side = math.sqrt(c["n"])
    m = _model(c["n"], side, seed + 1, c["relax"])
    p = ParameterArrays(m.num(), erodibility=_lognormal(m.num(), seed + 2),
                        is_outlet=_border(m, side) if c["outlets"] == "border" else False,
                        max_slope=SLOPE if c["slope"] else None)
    return m, p


def _sizes(c, count):
    """Site counts spread evenly over the logarithm of [lo, hi], large and small in turn."""
    ns = [int(c["lo"] * (c["hi"] / c["lo"]) ** (i / max(1, count - 1))) for i in range(count)]
    return [ns[i // 2] if i % 2 else ns[count - 1 - i // 2] for i in range(count)]


def _many(c, count, seed):
    """`count` terrains of the sizes above, outlets along the border."""
    from concurrent.futures import ThreadPoolExecutor
    ns = _sizes(c, count)
    with ThreadPoolExecutor(16) as ex:
        ms = list(ex.map(lambda i: _model(ns[i], math.sqrt(ns[i]), seed * 64 + i + 1), range(count)))
    ps = [ParameterArrays(m.num(), erodibility=_lognormal(m.num(), seed * 64 + i),
                          is_outlet=_border(m, math.sqrt(m.num()))) for i, m in enumerate(ms)]
    return ms, ps


def _lattice(w, h, seed):
    """A w x h height-map lattice: jittered sites, each quad cut along one of its two
    diagonals, rows listing the neighbours counter-clockwise from the east."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    g = torch.Generator(device=dev).manual_seed(seed)
    n = w * h
    x = (torch.arange(w, device=dev, dtype=torch.float64)[None, :]
         + torch.rand((h, w), generator=g, device=dev, dtype=torch.float64) * 0.6 - 0.3)
    y = (torch.arange(h, device=dev, dtype=torch.float64)[:, None]
         + torch.rand((h, w), generator=g, device=dev, dtype=torch.float64) * 0.6 - 0.3)
    # quad (i, j) between rows i, i + 1 and columns j, j + 1: True cuts it from (i, j) to
    # (i + 1, j + 1)
    up = torch.rand((h - 1, w - 1), generator=g, device=dev) < 0.5
    area = 0.5 + torch.rand((h, w), generator=g, device=dev, dtype=torch.float64)
    k = 0.2 + 1.6 * torch.rand((h, w), generator=g, device=dev, dtype=torch.float64)
    steps = [(0, 1), (1, 1), (1, 0), (1, -1), (0, -1), (-1, -1), (-1, 0), (-1, 1)]
    has = torch.zeros((8, h, w), device=dev, dtype=torch.bool)
    has[0][:, :-1] = True
    has[4][:, 1:] = True
    has[2][:-1] = True
    has[6][1:] = True
    has[1][:-1, :-1] = up
    has[5][1:, 1:] = up
    has[3][:-1, 1:] = ~up
    has[7][1:, :-1] = ~up
    row = torch.zeros(n + 1, device=dev, dtype=torch.int64)
    row[1:] = torch.cumsum(has.sum(0).reshape(-1), 0)
    flat = has.permute(1, 2, 0).reshape(n, 8)
    del has
    ids = torch.arange(n, device=dev, dtype=torch.int32)[:, None]
    off = torch.tensor([dy * w + dx for dy, dx in steps], device=dev, dtype=torch.int32)[None, :]
    col = (ids + off)[flat]
    src = ids.expand(n, 8)[flat]
    del flat
    x, y = x.reshape(-1), y.reshape(-1)
    ln = torch.sqrt((x[col] - x[src]) ** 2 + (y[col] - y[src]) ** 2)
    outlet = torch.zeros((h, w), device=dev, dtype=torch.uint8)
    outlet[0, :] = outlet[:, 0] = 1                        # two sides of the map drain
    a = lambda t, dt: t.reshape(-1).to(dt).cpu().numpy()
    m = TerrainModel2D(a(x, torch.float64), a(y, torch.float64), a(area, torch.float64),
                       row.to(torch.int32).cpu().numpy().view(np.uint32),
                       col.cpu().numpy().view(np.uint32), ln.cpu().numpy(),
                       np.arange(w, dtype=np.uint32))
    p = ParameterArrays(n, erodibility=a(k, torch.float64), is_outlet=a(outlet, torch.uint8)).pinned()
    return m, p


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "solve":
        m, p = _solve_inputs(c, seed)
        m.handle()
        return {"case": c, "m": m, "p": p}
    if kind == "grid":
        m, p = _lattice(c["w"], c["h"], seed + 1)
        m.handle()
        return {"case": c, "m": m, "p": p, "out": pinned_empty(m.num(), np.float64)}
    if kind == "fresh":
        m, p = _solve_inputs(dict(c, relax=0, slope=False, outlets="border"), seed)
        return {"case": c, "m": m, "p": p}
    if kind == "batch":
        ms, ps = _many(c, c["terrains"], seed + 1)
        b = TerrainBatch(ms)
        b.handle()
        return {"case": c, "b": b, "p": ps}
    if kind == "served":
        ms, ps = _many(c, c["requests"], seed + 1)
        s = TerrainServer(hbm_budget_bytes=40 * 10**9, slots=12)
        return {"case": c, "s": s, "ids": [s.add_model(m) for m in ms], "p": ps}
    side = math.sqrt(c["n"])
    rng = np.random.default_rng(seed + 3)
    b = TerrainModel2DBulider.from_random_sites(c["n"], Site2D(0.0, 0.0), Site2D(side, side), seed=seed + 1)
    e = rng.uniform(0.0, 500.0, c["n"])
    it = TerrainInterpolator2D(b.xs, b.ys)
    if kind == "profile":
        q = rng.uniform(0.05 * side, 0.95 * side, (2, c["queries"]))
        return {"case": c, "t": Terrain2D(b.xs, b.ys, e, interpolator=it), "qx": q[0].copy(), "qy": q[1].copy()}
    axis = (torch.arange(c["px"], device="cuda", dtype=torch.float64) + 0.5) * (side / c["px"])
    qy, qx = torch.meshgrid(axis, axis, indexing="ij")
    qx, qy = qx.reshape(-1).contiguous(), qy.reshape(-1).contiguous()
    return {"case": c, "it": it, "e": torch.from_numpy(e).cuda(), "qx": qx, "qy": qy,
            "out": torch.empty_like(qx), "found": torch.empty(qx.numel(), device="cuda", dtype=torch.uint8)}


def run(state):
    c = state["case"]
    kind, iters = c["kind"], c.get("iters", 0)
    if kind in ("solve", "grid", "fresh"):
        g = TerrainGenerator.default().set_model(state["m"]).set_parameters(state["p"])
        if iters:
            g.set_max_iteration(iters)
        t = g.generate(out=state.get("out"))
        if kind == "fresh":
            state["m"].release()
        return {"elevations": t.elevations(), "iterations": g.last_iterations}
    if kind == "batch":
        g = BatchGenerator().set_batch(state["b"]).set_parameters(state["p"])
        if iters:
            g.set_max_iteration(iters)
        ts = g.generate()
        return {"elevations": [t.elevations() for t in ts], "iterations": g.last_terrain_iterations}
    if kind == "served":
        s = state["s"]
        tickets = [s.submit(i, p, max_iteration=iters or None) for i, p in zip(state["ids"], state["p"])]
        done = [s.wait(t) for t in tickets]
        return {"elevations": [t.elevations() for t, _ in done],
                "iterations": np.array([info["iterations"] for _, info in done])}
    if kind == "profile":
        return {"elevations": state["t"].get_elevations(state["qx"], state["qy"], gpu=True)}
    state["it"].interpolate_device(state["e"], state["qx"], state["qy"], state["out"], state["found"])
    return {"elevations": state["out"], "found": state["found"]}


# ---- what a pass cannot do without ---------------------------------------------------

def _iterations(n, iters):
    """A terrain's iterations: about 0.334 n^0.565 until nothing changes (151 at 50,000 sites,
    327 at 200,000, 821 at 1,000,000), or the bound."""
    free = max(8.0, 0.334 * n**0.565)
    return min(free, iters) if iters else free


def _solve_work(n, iters):
    # an iteration reads per site its row pointer, cell area, elevation, erodibility, uplift and
    # outlet flag and per neighbour (six) a column and a length, and writes an elevation; its
    # operations are a difference and a quotient per neighbour, and the sums, root, product and
    # quotients of the area, time and elevation
    it = _iterations(n, iters)
    return {"bytes": n * it * (45 + 12 * 6) + 33 * n, "flops": n * it * (2 * 6 + 10)}


def work(case):
    c, kind = case, case["kind"]
    if kind == "grid":
        return _solve_work(c["w"] * c["h"], c["iters"])
    if kind == "solve":
        return _solve_work(c["n"], c["iters"])
    if kind == "fresh":
        w = _solve_work(c["n"], c["iters"])
        return {"bytes": w["bytes"] + c["n"] * (28 + 12 * 6), "flops": w["flops"]}
    if kind in ("batch", "served"):
        count = c["terrains"] if kind == "batch" else c["requests"]
        ws = [_solve_work(n, c["iters"]) for n in _sizes(c, count)]
        return {"bytes": sum(w["bytes"] for w in ws), "flops": sum(w["flops"] for w in ws)}
    # a query reads its point and writes a value and a flag; the sites, their values and the
    # triangles (two a site) are read once; about six neighbours take some 40 operations each
    q = c["queries"] if kind == "profile" else c["px"] ** 2
    return {"bytes": q * 25 + min(c["n"], 8 * q) * (24 + 2 * 24), "flops": q * 6 * 40}


# ---- the same results from numpy ------------------------------------------------------

def _noise(n):
    """n draws of gen::<f64>() from the generator's StdRng (ChaCha12, seed_from_u64(0))."""
    state, key = 0, []
    for _ in range(8):
        state = (state * 6364136223846793005 + 11634580027462260723) % 2**64
        x = (((state >> 18) ^ state) >> 27) % 2**32
        r = state >> 59
        key.append(((x >> r) | (x << ((32 - r) % 32))) % 2**32)
    blocks = (n + 7) // 8
    words = [0x61707865, 0x3320646E, 0x79622D32, 0x6B206574] + key + [None, 0, 0, 0]
    init = [np.arange(blocks, dtype=np.uint32) if v is None else np.full(blocks, v, np.uint32) for v in words]
    s = [v.copy() for v in init]
    rot = lambda v, k: (v << np.uint32(k)) | (v >> np.uint32(32 - k))

    def quarter(a, b, c, d):
        s[a] = s[a] + s[b]
        s[d] = rot(s[d] ^ s[a], 16)
        s[c] = s[c] + s[d]
        s[b] = rot(s[b] ^ s[c], 12)
        s[a] = s[a] + s[b]
        s[d] = rot(s[d] ^ s[a], 8)
        s[c] = s[c] + s[d]
        s[b] = rot(s[b] ^ s[c], 7)

    for _ in range(6):
        for i in range(4):
            quarter(i, 4 + i, 8 + i, 12 + i)
        for i in range(4):
            quarter(i, 4 + (i + 1) % 4, 8 + (i + 2) % 4, 12 + (i + 3) % 4)
    out = np.stack([a + b for a, b in zip(s, init)], 1).astype(np.uint64).reshape(-1)
    bits = (out[0::2] | (out[1::2] << np.uint64(32)))[:n]
    return (bits >> np.uint64(11)).astype(np.float64) * 2.0**-53


def _pop_order(m, outlets):
    """The order in which a binary max-heap on the reversed edge length (std's BinaryHeap: ties
    by position) takes the sites, from the outlets at key 0."""
    heap, seen, rank = [], np.zeros(m.n, bool), np.full(m.n, m.n, np.int64)
    row, col, ln = m.row_ptr.tolist(), m.col.tolist(), m.length.tolist()

    def rise(item, pos):
        while pos > 0 and item[1] < heap[(pos - 1) >> 1][1]:
            heap[pos] = heap[(pos - 1) >> 1]
            pos = (pos - 1) >> 1
        heap[pos] = item

    def push(item):
        heap.append(item)
        rise(item, len(heap) - 1)

    for o in outlets:
        push((o, 0.0))
    count = 0
    while heap:
        last = heap.pop()
        v = last[0]
        if heap:
            v, pos, end = heap[0][0], 0, len(heap)
            while 2 * pos + 2 < end:           # down to a leaf along the nearer children
                child = 2 * pos + 1
                if not heap[child + 1][1] > heap[child][1]:
                    child += 1
                heap[pos] = heap[child]
                pos = child
            if 2 * pos + 2 == end:
                heap[pos] = heap[2 * pos + 1]
                pos = 2 * pos + 1
            rise(last, pos)
        if seen[v]:
            continue
        seen[v] = True
        rank[v] = count
        count += 1
        for s in range(row[v], row[v + 1]):
            if not seen[col[s]]:
                push((col[s], ln[s]))
    return rank


def _reference(m, p, iters):
    """generate() in numpy: (elevations, iterations)."""
    n, row, col, ln = m.n, m.row_ptr.astype(np.int64), m.col.astype(np.int64), m.length
    src = np.repeat(np.arange(n), np.diff(row))
    outlets = np.flatnonzero(p.is_outlet)
    if not len(outlets):
        outlets = m.default_outlets.astype(np.int64)
    is_out = np.zeros(n, bool)
    is_out[outlets] = True
    tan = None if p.max_slope is None else np.tan(p.max_slope)
    elev = p.base + _noise(n) * 2.0**-52
    rank = None
    done = 0
    while not iters or done < iters:
        done += 1
        with np.errstate(invalid="ignore"):
            slope = np.where(elev[src] > elev[col], (elev[src] - elev[col]) / ln, 0.0)
        top = np.maximum.reduceat(slope, row[:-1])
        best = np.flatnonzero((slope == top[src]) & (slope > 0) & ~is_out[src])
        nxt = np.arange(n)
        nxt[src[best[::-1]]] = col[best[::-1]]              # the first of equals is written last
        root = nxt
        while True:
            up = root[root]
            if np.array_equal(up, root):
                break
            root = up
        if not is_out[root].all():
            if rank is None:
                rank = _pop_order(m, outlets.tolist())
            lake = root[col]
            s = np.flatnonzero(~is_out[lake] & (lake != root[src]) & (rank[src] < n))
            s = s[np.lexsort((s, rank[src[s]]))]
            lakes, first = np.unique(lake[s], return_index=True)
            for slot in s[first].tolist():
                k, nk = int(col[slot]), int(src[slot])
                while nxt[k] != k:
                    nxt[k], nk, k = nk, k, int(nxt[k])
                nxt[k] = nk
        dist = np.ones(n)
        edge = nxt[src] == col
        dist[src[edge][::-1]] = ln[edge][::-1]
        # sites by level below the roots, receivers before donors
        donors = np.flatnonzero((nxt[col] == src) & (col != src))     # slots (receiver, donor)
        start = np.searchsorted(src[donors], np.arange(n + 1))
        level, frontier = [], np.flatnonzero(nxt == np.arange(n))
        slots_of = []
        while len(frontier):
            level.append(frontier)
            cnt = start[frontier + 1] - start[frontier]
            take = np.repeat(start[frontier], cnt) + np.arange(cnt.sum()) - np.repeat(np.cumsum(cnt) - cnt, cnt)
            slots_of.append(donors[take])
            frontier = col[donors[take]]
        area = m.area.copy()
        for d in range(len(level) - 1, -1, -1):
            s = slots_of[d][::-1]
            np.add.at(area, src[s], area[col[s]])
        w = 1.0 / (p.erodibility * np.sqrt(area)) * dist
        t, new = np.zeros(n), elev.copy()
        out_t, out_e = np.zeros(n), np.zeros(n)
        for d, v in enumerate(level):
            r = nxt[v]
            t[v] = (t[r] if d else 0.0) + w[v]
            out_t[v] = out_t[r] if d else t[v]
            out_e[v] = out_e[r] if d else elev[v]
            e = out_e[v] + p.uplift[v] * np.maximum(t[v] - out_t[v], 0.0)
            if tan is not None and d:
                steep = (e - new[r]) / dist[v] > tan[v]
                e = np.where(steep, new[r] + tan[v] * dist[v], e)
            new[v] = e
        same = np.array_equal(new, elev)
        elev = new
        if same:
            break
    return elev, done


def _clip(poly, a, b, c):
    """The part of a polygon with a x + b y <= c."""
    out = []
    for i, (x, y) in enumerate(poly):
        u, v = poly[i - 1]
        f, g = a * x + b * y - c, a * u + b * v - c
        if (f <= 0.0) != (g <= 0.0):
            r = g / (g - f)
            out.append((u + (x - u) * r, v + (y - v) * r))
        if f <= 0.0:
            out.append((x, y))
    return out


def _nearer(poly, p, q):
    """The part of a polygon nearer to p than to q."""
    dx, dy = q[0] - p[0], q[1] - p[1]
    return _clip(poly, dx, dy, dx * 0.5 * (p[0] + q[0]) + dy * 0.5 * (p[1] + q[1]))


def _area(poly):
    x0, y0 = poly[0]
    return 0.5 * abs(sum((poly[i - 1][0] - x0) * (poly[i][1] - y0) - (poly[i][0] - x0) * (poly[i - 1][1] - y0)
                         for i in range(len(poly))))


def _sibson(xs, ys, e, qx, qy):
    """Each query's mean of its natural neighbours' values, weighted by the area its cell takes
    from theirs; the queries lie inside the hull."""
    out, span = np.empty(len(qx)), 100.0 * float(xs.max() - xs.min())
    for i, q in enumerate(zip(qx.tolist(), qy.tolist())):
        d2 = (xs - q[0]) ** 2 + (ys - q[1]) ** 2
        near = np.argpartition(d2, 64)[:64] if len(xs) > 256 else np.arange(len(xs))
        near = near[np.argsort(d2[near])]
        while True:
            cell = [(q[0] - span, q[1] - span), (q[0] + span, q[1] - span), (q[0] + span, q[1] + span), (q[0] - span, q[1] + span)]
            for j in near.tolist():
                reach = 4.0 * max((x - q[0]) ** 2 + (y - q[1]) ** 2 for x, y in cell)
                if d2[j] > reach:
                    break
                cell = _nearer(cell, q, (float(xs[j]), float(ys[j])))
            reach = 4.0 * max((x - q[0]) ** 2 + (y - q[1]) ** 2 for x, y in cell)
            if len(near) == len(xs) or d2[near[-1]] > reach:
                break
            near = np.argsort(d2)
        rival = [(float(xs[j]), float(ys[j]), float(e[j])) for j in near.tolist() if d2[j] <= reach]
        total = value = 0.0
        for a in rival:
            part = cell
            for b in rival:
                if b is not a:
                    part = _nearer(part, a, b)
                    if len(part) < 3:
                        break
            if len(part) >= 3:
                w = _area(part)
                total += w
                value += w * a[2]
        out[i] = value / total
    return out


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "solve" and c["n"] * _iterations(c["n"], c["iters"]) < 1.3e7:
        m, p = _solve_inputs(c, seed)
        e, it = _reference(m, p, c["iters"])
        return {"elevations": e, "iterations": it}
    if kind == "fresh" and c["n"] * c["iters"] < 1.3e7:
        m, p = _solve_inputs(dict(c, relax=0, slope=False, outlets="border"), seed)
        e, it = _reference(m, p, c["iters"])
        return {"elevations": e, "iterations": it}
    if kind == "profile" and c["queries"] <= 4000:
        side = math.sqrt(c["n"])
        rng = np.random.default_rng(seed + 3)
        b = TerrainModel2DBulider.from_random_sites(c["n"], Site2D(0.0, 0.0), Site2D(side, side), seed=seed + 1)
        e = rng.uniform(0.0, 500.0, c["n"])
        q = rng.uniform(0.05 * side, 0.95 * side, (2, c["queries"]))
        return {"elevations": _sibson(b.xs, b.ys, e, q[0], q[1])}
    return None
