"""The work that the engine's timings are taken on: joins of synthetic parcel layers through the Python binding.

The layers are the seeded Voronoi tilings of gsj.gen, whose distributions the benchmark, the tests and the serving
schedule use: parcels of 4-256 vertices per ring (log-uniform, 5% multipolygons, 2% holes), parcels of ~30 vertices,
zones, large polygons of thousands of vertices. The parcel density is the benchmark's (500k per square degree), so a
layer's box follows from its size. prepare() makes host layers from the seed and uploads them (layers and their trees stay
resident in a user's program); run() is one call of the engine and returns its rows.

The polygon joins hand their rows over in no set order; run() puts them in the order of their ids on the device, as a
program that merges or writes them does.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "postgis-cuda_b200"))
import gsj  # noqa: E402
from gsj import gen  # noqa: E402

X0, Y0, DENSITY = -119.0, 33.0, 500_000.0

# mean vertices of a geometry of each kind of layer (closing vertices included)
NV = {"parcels": 68.0, "query": 107.0, "cfg5": 34.6, "zones": 24.4, "wide": 6.0}


def listed():
    return [
        # the smallest request of the serving stream: 100 query polygons against a resident layer, intersects + area; latency counts
        {"name": "request_area_100", "op": "request", "want": "area", "n": 100, "m": 200_000},
        # the plain intersects + area join: 20k small zones by 50 wide ones
        {"name": "zones_area", "op": "zones", "n": 20_000, "m": 50},
        # an ordinary relate request of the serving stream
        {"name": "request_relate_20k", "op": "request", "want": "relate", "n": 20_011, "m": 200_000},
        # the headline: DE-9IM relate of a parcel layer with itself, each unordered pair once
        {"name": "parcels_relate", "op": "self", "want": "relate", "n": 500_000},
        # parcels by the parcels of another source: the interiors overlap, every pair has an area
        {"name": "layers_area", "op": "layers", "want": "area", "n": 120_000, "m": 120_000},
        # parcels by polygons of 2000-8000 vertices that LOAD subdivided at 256: the piece pairs are folded
        {"name": "subdivided_area", "op": "subdivided", "n": 60_000, "m": 50},
        # addresses in parcels
        {"name": "points_in_parcels", "op": "pip", "n": 1_000_000, "m": 200_000},
        # addresses within 5 m of parcels on the spheroid
        {"name": "points_dwithin", "op": "points_dwithin", "d": 5.0, "n": 1_000_000, "m": 200_000},
        # parcels within 5 m of each other on the spheroid
        {"name": "parcels_dwithin", "op": "dwithin", "d": 5.0, "n": 150_000},
        # parcels that still meet when each is shrunk by 1 m (negative buffer), self pairs kept
        {"name": "parcels_erode", "op": "erode", "d": 1.0, "n": 200_000, "two": False},
        # connected components of parcels that meet, many components of every size
        {"name": "parcels_cluster", "op": "cluster", "n": 300_000},
        # one-shot use: a host layer is uploaded (tree built) and joined with itself, then dropped
        {"name": "load_relate", "op": "load", "want": "relate", "n": 200_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["request", "request", "zones", "self", "layers", "subdivided", "pip", "points_dwithin", "dwithin", "erode", "cluster", "load"])
    if op == "request":
        return {"op": op, "want": rng.choice(["area", "relate", "dwithin"]), "n": _log(rng, 100, 30_000), "m": _log(rng, 50_000, 200_000)}
    if op == "zones":
        return {"op": op, "n": _log(rng, 2_000, 50_000), "m": _log(rng, 20, 200)}
    if op == "self":
        return {"op": op, "want": rng.choice(["relate", "area", "both"]), "n": _log(rng, 5_000, 300_000)}
    if op == "layers":
        return {"op": op, "want": rng.choice(["area", "relate", "both"]), "n": _log(rng, 5_000, 100_000), "m": _log(rng, 5_000, 100_000)}
    if op == "subdivided":
        return {"op": op, "n": _log(rng, 5_000, 60_000), "m": _log(rng, 10, 100)}
    if op == "pip":
        return {"op": op, "n": _log(rng, 20_000, 1_000_000), "m": _log(rng, 20_000, 200_000)}
    if op == "points_dwithin":
        return {"op": op, "d": rng.choice([1.0, 5.0, 20.0]), "n": _log(rng, 20_000, 500_000), "m": _log(rng, 20_000, 200_000)}
    if op == "dwithin":
        return {"op": op, "d": rng.choice([1.0, 5.0, 20.0]), "n": _log(rng, 5_000, 100_000)}
    if op == "erode":
        two = rng.random() < 0.5
        return {"op": op, "d": rng.choice([1.0, 4.0]), "n": _log(rng, 5_000, 60_000 if two else 150_000), "two": two}
    if op == "cluster":
        return {"op": op, "n": _log(rng, 10_000, 300_000)}
    return {"op": op, "want": "relate", "n": _log(rng, 5_000, 200_000)}


# ---- inputs ------------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _engine():
    return gsj.Engine(0)   # a program has one context and keeps it


def _box(n, x0=X0, y0=Y0):
    side = math.sqrt(n / DENSITY)
    return (x0, y0, x0 + side, y0 + side)


def _outer(b):
    """A box a little larger on every side: layers of two sources share no border line (on a shared one a long edge meets more collinear edges
    than the eight intervals that the reference's rules keep per edge)."""
    w, h = b[2] - b[0], b[3] - b[1]
    return (b[0] - 0.011 * w, b[1] - 0.013 * h, b[2] + 0.017 * w, b[3] + 0.007 * h)


def _host(case, seed):
    """The host layers of a case: (P, R); R is P for a layer joined with itself; points are an (n, 2) array."""
    s, op, n = 2 * int(seed) + 1, case["op"], case["n"]
    m = case.get("m", n)
    if op == "request":   # queries as the serving schedule draws them: a window of the resident layer at its density
        r = np.random.default_rng(s)
        big, side = math.sqrt(m / DENSITY), math.sqrt(n / DENSITY)
        qb = _box(n, X0 + r.uniform(0, max(big - side, 0)), Y0 + r.uniform(0, max(big - side, 0)))
        return (gen.voronoi(n, qb, s, jitter_grid=True, jitter=0.4, vmin=4, vmax=512, log_uniform=True), gen.layer_parcels(m, _box(m), s + 1))
    if op == "zones":
        return gen.layer_cfg_parcels_small(n, s), gen.voronoi(m, _outer(gen.LA_BOX), s + 1, vmin=4, vmax=4)
    if op in ("self", "load", "dwithin"):
        p = gen.layer_parcels(n, _box(n), s)
        return p, p
    if op == "layers":   # the same box for both, so n and m also set how much larger one side's geometries are
        b = _box(max(n, m))
        return gen.layer_parcels(n, b, s), gen.layer_parcels(m, _outer(b), s + 1)
    if op == "subdivided":
        b = _box(n)
        return gen.layer_parcels(n, b, s), gen.voronoi(m, _outer(b), s + 1, vmin=2000, vmax=8000)
    if op in ("pip", "points_dwithin"):
        return gen.points(n, _box(m), s), gen.layer_parcels(m, _box(m), s + 1)
    if op == "erode":
        p = gen.layer_cfg5(n, _box(n), s)
        return p, gen.layer_cfg5(n, _outer(_box(n)), s + 1) if case["two"] else p
    if op == "cluster":
        p = gen.shrunk(gen.layer_cfg5(n, _box(n), s), s)
        return p, p
    raise ValueError(op)


def _pinned(a):
    t = torch.empty(a.size, dtype=torch.int64 if a.dtype == np.uint64 else torch.float64, pin_memory=True)
    v = t.numpy().view(a.dtype).reshape(a.shape)
    v[...] = a
    return v


def _capacity(case):
    """Rows that the result table of a case holds; a tiling's row count varies a little from seed to seed."""
    n, m, op = case["n"], case.get("m", case["n"]), case["op"]
    per = {"request": 6, "zones": 2, "self": 5, "load": 5, "subdivided": 2, "pip": 2, "points_dwithin": 3, "dwithin": 8, "cluster": 1}
    if op == "layers":
        return int(1.8 * (math.sqrt(n) + math.sqrt(m)) ** 2) + 2000
    return (per[op] if op in per else 7 if case["two"] else 2) * n + 2000


def prepare(case, seed):
    eng, (p, r) = _engine(), _host(case, seed)
    st = {"case": case, "eng": eng, "table": _table(case)}
    if case["op"] == "load":   # the arrays of a loader that reads into pinned memory
        st["host"] = gen.PolygonSet(_pinned(p.gro), _pinned(p.rvo), _pinned(p.xy))
        return st
    if case["op"] == "subdivided":
        r = eng.subdivide(r, 256)
    st["P"] = eng.upload_points(p) if isinstance(p, np.ndarray) else eng.upload_polygons(p)
    st["R"] = st["P"] if r is p else eng.upload_polygons(r)
    return st


def _table(case, dev="cuda"):
    """The device result table of a program that takes the rows on: a column per kind of value; unused rows at the end
    are -1, their areas 0."""
    op, want, cap = case["op"], case.get("want", "area"), _capacity(case)
    polygons = op in ("request", "zones", "self", "layers", "subdivided", "load") and want != "dwithin"
    cols = {"root": torch.int32} if op == "cluster" else {"pairs": torch.int64}
    if op == "pip":
        cols["where"] = torch.uint8
    if polygons and want in ("area", "both"):
        cols["area"] = torch.float64
    if polygons and want in ("relate", "both"):
        cols["code"] = torch.int32
    return {k: torch.empty(cap, dtype=t, device=dev) for k, t in cols.items()}


def _fill(table, cols):
    for k, v in cols.items():
        t, n = table[k], len(v)
        if n > len(t):
            raise RuntimeError(f"{n} rows: the table holds {len(t)}")
        t[:n] = v
        t[n:] = 0 if t.dtype == torch.float64 else 255 if t.dtype == torch.uint8 else -1
    return table


def _ids(pairs):
    return torch.from_numpy(pairs.view(np.int64).reshape(-1))


def _rows(table, r):
    """The rows of a polygon join, ordered by their ids on the device."""
    key, at = _ids(r.pairs).cuda().sort()
    cols = {"pairs": key}
    if r.area is not None:
        cols["area"] = torch.from_numpy(r.area).cuda()[at]
    if r.code is not None:
        cols["code"] = torch.from_numpy(r.code.view(np.int32)).cuda()[at]
    return _fill(table, cols)


def run(st):
    c, eng, table = st["case"], st["eng"], st["table"]
    op, want = c["op"], c.get("want", "area")
    flags = {"want_area": want in ("area", "both"), "want_relate": want in ("relate", "both")}
    if op == "load":
        lay = eng.upload_polygons(st["host"])
        out = _rows(table, eng.join(lay, lay, upper=True, **flags))
        lay.free()
        return out
    P, R = st["P"], st["R"]
    if op == "request" and want == "dwithin":
        return _fill(table, {"pairs": _ids(eng.dwithin(P, R, 5.0)[0])})
    if op in ("request", "zones", "self", "layers", "subdivided"):
        return _rows(table, eng.join(P, R, upper=P is R, **flags))
    if op == "pip":
        pairs, where, _ = eng.join_points(P, R)
        return _fill(table, {"pairs": _ids(pairs), "where": torch.from_numpy(where)})
    if op == "points_dwithin":
        return _fill(table, {"pairs": _ids(eng.points_dwithin(P, R, c["d"])[0])})
    if op == "dwithin":
        return _fill(table, {"pairs": _ids(eng.dwithin(P, P, c["d"], same=True)[0])})
    if op == "erode":
        return _fill(table, {"pairs": _ids(eng.erode(P, R, c["d"], c["d"], same=P is R)[0])})
    return _fill(table, {"root": torch.from_numpy(eng.cluster(P)[0].view(np.int32))})


# ---- what a pass cannot do without ---------------------------------------------------------------------------------
def work(case):
    """bytes: each layer's vertices (16 bytes) and boxes (16 bytes) read once, each row written once; flops: per result pair,
    one classification (70 FP64 operations: four orientations and one boundary term) of each edge of the two that lies near the other (about
    half of a geometry's edges in a tiling; for points one crossing test of 12 operations per edge)."""
    op, n = case["op"], case["n"]
    m, want = case.get("m", n), case.get("want", "area")
    kinds = {"request": ("query", "parcels"), "zones": ("zones", "wide"), "layers": ("parcels", "parcels"), "subdivided": ("parcels", "parcels")}
    va, vb = (NV[k] for k in kinds.get(op, ("cfg5", "cfg5") if op in ("erode", "cluster") else ("parcels", "parcels")))
    row = 8 + (8 if want in ("area", "both") else 0) + (4 if want in ("relate", "both") else 0)
    if op in ("pip", "points_dwithin"):
        rows = 1.2 * n
        return {"bytes": n * 16 + m * (vb * 16 + 16) + rows * (9 if op == "pip" else 8), "flops": rows * vb * 12}
    one = op in ("self", "load", "dwithin", "cluster") or (op == "erode" and not case["two"])
    if op == "request":   # only the part of the resident layer under the window
        m = min(m, 1.3 * n)
    if op == "subdivided":
        layer = n * (va * 16 + 16) + m * 4400 * 16
        rows = 1.15 * n
        vb = 0.2 * va
    elif op == "zones":
        layer = n * (va * 16 + 16) + m * (vb * 16 + 16)
        rows, vb = 1.1 * n, vb
    else:
        layer = n * (va * 16 + 16) + (0 if one else m * (vb * 16 + 16))
        rows = 3.8 * n if one else 4.6 * max(n, m)
    if op == "cluster":   # a spanning forest's pairs have to be tested, and each geometry's label written
        return {"bytes": layer + 4 * n, "flops": n * (va + vb) * 0.5 * 70}
    if op in ("dwithin", "erode"):
        row = 8
    out = n if op == "erode" and one else rows
    return {"bytes": layer + out * row, "flops": rows * (va + vb) * 0.5 * 70}


def tolerance(case):
    """Pairs, DE-9IM codes, positions and labels are whole numbers. Areas: sums of FP64 cross products near 0 in a pair's frame; an
    implementation that contracts multiply-adds was measured 2.3e-10 away."""
    return {"rel": 1e-9} if _has_area(case) else "exact"


def _has_area(case):
    return case["op"] in ("zones", "subdivided") or (case["op"] in ("request", "self", "layers") and case["want"] in ("area", "both"))


# ---- intersection areas in 64 bits, without the engine ---------------------------------------------------------------
def _ring_edges(ps, dev):
    """All edges of a layer: x0, y0, x1, y1 (relative to the box corner), the first edge of each geometry, boxes."""
    xy = torch.from_numpy(ps.xy).to(dev) - torch.tensor([X0, Y0], dtype=torch.float64, device=dev)
    rvo = torch.from_numpy(ps.rvo.astype(np.int64)).to(dev)
    last = torch.zeros(len(xy), dtype=torch.bool, device=dev)
    last[rvo[1:] - 1] = True
    first_v = rvo[torch.from_numpy(ps.gro.astype(np.int64)).to(dev)]
    keep = torch.nonzero(~last).reshape(-1)
    off = torch.searchsorted(keep, first_v)
    e = torch.stack([xy[keep, 0], xy[keep, 1], xy[keep + 1, 0], xy[keep + 1, 1]])
    v0 = ps.rvo[ps.gro[:-1]].astype(np.int64)
    lo = torch.from_numpy(np.minimum.reduceat(ps.xy, v0, axis=0) - np.array([X0, Y0])).to(dev)
    hi = torch.from_numpy(np.maximum.reduceat(ps.xy, v0, axis=0) - np.array([X0, Y0])).to(dev)
    return e, off, lo, hi


def _spread(start, count):
    """For each i its count[i] numbers start[i], start[i] + 1, ...: (which i, number)."""
    which = torch.repeat_interleave(torch.arange(len(count), device=count.device), count)
    first = torch.cumsum(count, 0) - count
    return which, start[which] + torch.arange(len(which), device=count.device) - first[which]


def _chunks(cost, most):
    edge = torch.cumsum(cost, 0)
    at = 0
    while at < len(cost):
        base = int(edge[at - 1]) if at else 0
        to = max(at + 1, int(torch.searchsorted(edge, base + most, right=True)))
        yield at, to
        at = to


def _areas(p, r, upper, dev):
    """(a, b, area) of the pairs that share area. Every polygon is the signed sum of the trapezoids between its edges and a base
    line, so the shared area is the signed sum over edge pairs of the integral of the lower edge above the base line."""
    ea, offa, loa, hia = _ring_edges(p, dev)
    eb, offb, lob, hib = (ea, offa, loa, hia) if r is p else _ring_edges(r, dev)
    pa, pb = [], []
    rows = max(1, 50_000_000 // len(lob))
    for i in range(0, len(loa), rows):
        l, h = loa[i:i + rows], hia[i:i + rows]
        k = (l[:, None, 0] < hib[None, :, 0]) & (h[:, None, 0] > lob[None, :, 0]) & (l[:, None, 1] < hib[None, :, 1]) & (h[:, None, 1] > lob[None, :, 1])
        x, y = torch.nonzero(k, as_tuple=True)
        pa.append(x + i)
        pb.append(y)
    pa, pb = torch.cat(pa), torch.cat(pb)
    if upper:
        k = pb >= pa
        pa, pb = pa[k], pb[k]
    base = torch.minimum(loa[pa, 1], lob[pb, 1])
    na, nb = (offa[1:] - offa[:-1])[pa], (offb[1:] - offb[:-1])[pb]
    area = torch.zeros(len(pa), dtype=torch.float64, device=dev)
    for s, t in _chunks(nb, 20_000_000):
        w, j = _spread(offb[pb[s:t]], nb[s:t])
        w = w + s
        bx0, bx1 = torch.minimum(eb[0, j], eb[2, j]), torch.maximum(eb[0, j], eb[2, j])
        k = (bx0 < hia[pa[w], 0]) & (bx1 > loa[pa[w], 0])   # b's edges under or over a
        w, j = w[k], j[k]
        for u, v in _chunks(na[w], 10_000_000):
            q, i = _spread(offa[pa[w[u:v]]], na[w[u:v]])
            q = q + u
            pair, jj = w[q], j[q]
            xl = torch.maximum(torch.minimum(ea[0, i], ea[2, i]), torch.minimum(eb[0, jj], eb[2, jj]))
            xr = torch.minimum(torch.maximum(ea[0, i], ea[2, i]), torch.maximum(eb[0, jj], eb[2, jj]))
            k = xr > xl
            xl, xr, pair, i, jj = xl[k], xr[k], pair[k], i[k], jj[k]
            f, g = ea[:, i], eb[:, jj]
            bl = base[pair]
            fa, ga = (f[3] - f[1]) / (f[2] - f[0]), (g[3] - g[1]) / (g[2] - g[0])
            fl, fr = f[1] - bl + (xl - f[0]) * fa, f[1] - bl + (xr - f[0]) * fa
            gl, gr = g[1] - bl + (xl - g[0]) * ga, g[1] - bl + (xr - g[0]) * ga
            dl, dr = fl - gl, fr - gr
            neg = torch.minimum(dl, dr)
            cross = (dl < 0) != (dr < 0)
            low = torch.where(cross, -0.5 * neg * neg / (dl - dr).abs().clamp_min(1e-300), 0.5 * (dl.clamp_max(0) + dr.clamp_max(0)))
            term = (0.5 * (gl + gr) + low) * (xr - xl)
            sign = torch.where(f[0] > f[2], 1.0, -1.0) * torch.where(g[0] > g[2], 1.0, -1.0)
            area.index_add_(0, pair, sign * term)
    k = area > 1e-13 * torch.minimum((hia - loa).prod(1)[pa], (hib - lob).prod(1)[pb])   # below: the rounding of the sum
    return pa[k], pb[k], area[k]


def exact(case, seed):
    """The areas of the pairs that share area; the pairs themselves have no computed value. A layer with itself also has rows of
    pairs that only touch, which a sum of areas does not show: no answer for it."""
    if not _has_area(case) or case["op"] == "self":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if dev == "cpu" and case["n"] > 5_000:
        return None
    p, r = _host(case, seed)
    a, b, area = _areas(p, r, False, dev)
    out = dict.fromkeys(_table(case, dev))
    out["area"] = _fill({"area": torch.empty(_capacity(case), dtype=torch.float64, device=dev)}, {"area": area[(b << 32 | a).argsort()]})["area"]
    return out
