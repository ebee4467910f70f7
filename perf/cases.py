"""The work that a user of this framework has it do, at the sizes it is used at.

Point-by-polygon joins (against a resident index, a batch of independent joins, a join whose index is built first, and
sums per polygon over host geometry arrays), distance and nearest joins both ways round, WKB decode, and the export of
a join's pairs as frame indexers.  Inputs follow the workloads of ``vibespatial_b200.testing.synthetic`` (stars,
building footprints around Gaussian or Zipf-weighted sites, polygons with holes and parts with points on and beside
their edges), generated on the GPU.  ``run`` makes one call (or the few calls that belong together) and returns its
whole result.  Joins write into the caller's pair buffers, as a C caller's do: the pairs fill a prefix of each buffer,
whose length is the call's result, and the rest keeps its -1.
"""
from __future__ import annotations

import ctypes
import math

import torch

import vibespatial_b200 as vsb
from vibespatial_b200 import _abi
from vibespatial_b200.geometry import GeometryArray

DEV = "cuda"
PREDICATES = {"within": _abi.PRED_WITHIN, "intersects": _abi.PRED_INTERSECTS, "bbox": _abi.PRED_BBOX,
              "touches": _abi.PRED_TOUCHES}
METHODS = {"learned": _abi.METHOD_LEARNED, "rtree": _abi.METHOD_RTREE}


# ---------------------------------------------------------------------------------------------------------- cases --
def listed():
    return [
        # a lookup of a few points in a few regions: latency only
        {"name": "join_star_1k", "kind": "join", "data": "star", "points": 1_003, "polygons": 10,
         "predicate": "intersects", "method": "learned"},
        # how many points each region contains and what they sum to: one high-level call on geometry arrays
        {"name": "aggregate_100k", "kind": "aggregate", "data": "star", "points": 100_000, "polygons": 1_000,
         "predicate": "contains"},
        # GPS fixes against a city's building footprints, index resident
        {"name": "join_utm_10m", "kind": "join", "data": "utm", "points": 10_000_000, "polygons": 100_000,
         "predicate": "within", "method": "learned"},
        # the largest: skewed points against a million footprints
        {"name": "join_zipf_50m", "kind": "join", "data": "zipf", "points": 50_000_000, "polygons": 1_000_000,
         "predicate": "within", "method": "learned"},
        # cadastral data: holes, multipolygons, points snapped onto and beside the edges
        {"name": "join_degenerate_4m", "kind": "join", "data": "degenerate", "points": 4_000_001, "polygons": 40_000,
         "predicate": "intersects", "method": "learned"},
        # many independent joins of very different sizes as one plan, pairs in row order
        {"name": "batch_32", "kind": "batch", "data": "star", "jobs": 32, "points": 1_000_000, "polygons": 20_000,
         "predicate": "within"},
        # polygons seen for the first time: the index is built for this one join
        {"name": "build_join_utm", "kind": "build_join", "data": "utm", "points": 1_000_000, "polygons": 100_000,
         "predicate": "within"},
        # everything within a distance of a footprint
        {"name": "dwithin_zipf_10m", "kind": "dwithin", "data": "zipf", "points": 10_000_000, "polygons": 200_000,
         "distance": 0.25},
        # each point's nearest footprint, with the distances
        {"name": "nearest_utm_4m", "kind": "nearest", "data": "utm", "points": 4_000_000, "polygons": 100_000},
        # each footprint's nearest points
        {"name": "nearest_polygons_100k", "kind": "nearest_polygons", "data": "zipf", "points": 2_000_000,
         "polygons": 100_000},
        # a GeoParquet file's two geometry columns, as bytes on the device
        {"name": "wkb_20m", "kind": "wkb", "data": "zipf", "points": 20_000_000, "polygons": 400_000},
        # a join's pairs made into the row indexers of how='left', with an attribute that has to agree
        {"name": "export_left_20m", "kind": "export", "pairs": 8_600_000, "points": 20_000_000, "polygons": 400_000,
         "how": "left", "attribute": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["aggregate", "join", "join", "join", "batch", "build_join", "dwithin", "nearest",
                       "nearest_polygons", "wkb", "export"])
    if kind == "aggregate":
        points = _log_int(rng, 2_000, 1_000_000)
        return {"kind": kind, "data": "star", "points": points, "polygons": _log_int(rng, 20, 5_000),
                "predicate": rng.choice(["intersects", "contains", "covers"])}
    if kind == "join":
        data = rng.choice(["star", "utm", "zipf", "degenerate"])
        least, most = {"star": ((1_000, 10), (2_000_000, 50_000)), "utm": ((200_000, 5_000), (10_000_000, 200_000)),
                       "zipf": ((200_000, 5_000), (50_000_000, 1_000_000)),
                       "degenerate": ((20_000, 500), (4_000_000, 40_000))}[data]
        return {"kind": kind, "data": data, "points": _log_int(rng, least[0], most[0]),
                "polygons": _log_int(rng, least[1], most[1]),
                "predicate": rng.choice(["within", "within", "intersects", "bbox" if data != "degenerate" else "touches"]),
                "method": rng.choice(["learned", "learned", "learned", "rtree"])}
    if kind == "batch":
        return {"kind": kind, "data": "star", "jobs": rng.randint(2, 32), "points": _log_int(rng, 20_000, 1_000_000),
                "polygons": _log_int(rng, 200, 20_000), "predicate": rng.choice(["within", "intersects"])}
    if kind == "build_join":
        return {"kind": kind, "data": rng.choice(["utm", "star", "zipf"]), "points": _log_int(rng, 200_000, 2_000_000),
                "polygons": _log_int(rng, 5_000, 200_000), "predicate": rng.choice(["within", "intersects"])}
    if kind == "dwithin":
        return {"kind": kind, "data": "zipf", "points": _log_int(rng, 50_000, 10_000_000),
                "polygons": _log_int(rng, 1_000, 200_000), "distance": round(rng.uniform(0.05, 0.25), 3)}
    if kind == "nearest":
        return {"kind": kind, "data": rng.choice(["utm", "zipf"]), "points": _log_int(rng, 20_000, 4_000_000),
                "polygons": _log_int(rng, 1_000, 100_000)}
    if kind == "nearest_polygons":
        return {"kind": kind, "data": "zipf", "points": _log_int(rng, 20_000, 2_000_000),
                "polygons": _log_int(rng, 1_000, 100_000)}
    if kind == "wkb":
        return {"kind": kind, "data": rng.choice(["zipf", "star"]), "points": _log_int(rng, 50_000, 20_000_000),
                "polygons": _log_int(rng, 1_000, 400_000)}
    points = _log_int(rng, 20_000, 20_000_000)
    return {"kind": "export", "pairs": int(points * rng.uniform(0.1, 0.6)), "points": points,
            "polygons": _log_int(rng, 1_000, 400_000), "how": rng.choice(["left", "inner", "right", "outer"]),
            "attribute": rng.random() < 0.5}


# --------------------------------------------------------------------------------------------------------- inputs --
class _Polygons:
    """A polygon SoA on the GPU: float64 x, y and int32 ring, part and geometry offsets."""

    def __init__(self, x, y, ring_sizes, rings_per_part=None, parts_per_geom=None):
        self.x, self.y = x.contiguous(), y.contiguous()
        one = torch.ones_like(ring_sizes) if rings_per_part is None else rings_per_part
        many = torch.ones_like(one) if parts_per_geom is None else parts_per_geom
        self.ring_off, self.part_off, self.geom_off = (_offsets(c) for c in (ring_sizes, one, many))

    def struct(self):
        return _abi.make_polygons(self.x, self.y, self.ring_off, self.part_off, self.geom_off)

    def host(self):
        return [t.cpu().numpy() for t in (self.x, self.y, self.ring_off, self.part_off, self.geom_off)]


def _offsets(counts):
    out = torch.zeros(counts.numel() + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(counts, 0, out=out[1:])
    return out.to(torch.int32)


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uniform(g, n, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(n, dtype=torch.float64, device=DEV, generator=g)


def _lognormal(g, n, median, sigma):
    return median * torch.exp(sigma * torch.randn(n, dtype=torch.float64, device=DEV, generator=g))


def _randint(g, lo, hi, n):
    return torch.randint(lo, hi, (n,), device=DEV, generator=g)


def _stars(g, n):
    """Star polygons in [0, 1000]^2: radius lognormal(ln 10, 0.5), 8 to 64 vertices (each count equally often),
    radial jitter U(0.6, 1)."""
    cx, cy, r = _uniform(g, n, 0, 1000), _uniform(g, n, 0, 1000), _lognormal(g, n, 10.0, 0.5)
    nv = 8 + torch.randperm(n, device=DEV, generator=g) % 57
    start = torch.cumsum(nv, 0) - nv
    owner = torch.repeat_interleave(torch.arange(n, device=DEV), nv)
    total = owner.numel()
    # angles ascending within each polygon: one sort of owner + angle / 2 pi
    turn = torch.sort(owner.double() + _uniform(g, total)).values - owner.double()
    rad = r[owner] * _uniform(g, total, 0.6, 1.0)
    vx = cx[owner] + rad * torch.cos(2 * math.pi * turn)
    vy = cy[owner] + rad * torch.sin(2 * math.pi * turn)
    x = torch.empty(total + n, dtype=torch.float64, device=DEV)
    y = torch.empty_like(x)
    at = torch.arange(total, device=DEV) + owner
    x[at], y[at] = vx, vy
    close = start + torch.arange(n, device=DEV) + nv
    x[close], y[close] = vx[start], vy[start]
    return _Polygons(x, y, nv + 1)


_TEMPLATES = (  # rectangle, L, T, U, cross; unit sides
    ((0, 0), (1, 0), (1, 1), (0, 1)),
    ((0, 0), (1, 0), (1, .4), (.4, .4), (.4, 1), (0, 1)),
    ((0, 0), (1, 0), (1, .35), (.65, .35), (.65, 1), (.35, 1), (.35, .35), (0, .35)),
    ((0, 0), (1, 0), (1, 1), (.7, 1), (.7, .35), (.3, .35), (.3, 1), (0, 1)),
    ((.35, 0), (.65, 0), (.65, .35), (1, .35), (1, .65), (.65, .65), (.65, 1), (.35, 1), (.35, .65), (0, .65),
     (0, .35), (.35, .35)),
)


def _footprints(g, cx, cy, side):
    """Rotated footprints around (cx, cy): sides lognormal with median ``side``, 4 to 12 vertices."""
    n = cx.numel()
    share = torch.tensor([0.4, 0.65, 0.77, 0.89], dtype=torch.float64, device=DEV)
    kind = torch.bucketize((torch.randperm(n, device=DEV, generator=g) + 0.5) / n, share)
    w, h, th = _lognormal(g, n, side, 0.5), _lognormal(g, n, side, 0.5), _uniform(g, n, 0, math.pi)
    sizes = torch.tensor([len(t) + 1 for t in _TEMPLATES], device=DEV)[kind]
    start = torch.cumsum(sizes, 0) - sizes
    x = torch.empty(int(sizes.sum()), dtype=torch.float64, device=DEV)
    y = torch.empty_like(x)
    c, s = torch.cos(th), torch.sin(th)
    for k, t in enumerate(_TEMPLATES):
        rows = torch.nonzero(kind == k).reshape(-1)
        ring = torch.tensor(t + t[:1], dtype=torch.float64, device=DEV) - 0.5
        lx, ly = ring[:, 0] * w[rows, None], ring[:, 1] * h[rows, None]
        at = start[rows, None] + torch.arange(len(t) + 1, device=DEV)
        x[at] = cx[rows, None] + lx * c[rows, None] - ly * s[rows, None]
        y[at] = cy[rows, None] + lx * s[rows, None] + ly * c[rows, None]
    return _Polygons(x, y, sizes)


def _around(g, n, centers, cumulative, sigma, lo, hi):
    site = torch.searchsorted(cumulative, _uniform(g, n)).clamp_(max=len(centers) - 1)
    out = []
    for k in (0, 1):
        v = centers[site, k]
        v += sigma * torch.randn(n, dtype=torch.float64, device=DEV, generator=g)
        out.append(v.clamp_(lo[k], hi[k]))
    return out


def _sites(g, sites, power, lo, extent):
    # away from the frame's edge, onto which the points beyond it are clamped
    centers = torch.stack([_uniform(g, sites, o + 0.08 * extent, o + 0.92 * extent) for o in lo], 1)
    w = 1.0 / torch.arange(1, sites + 1, dtype=torch.float64, device=DEV) ** power
    return centers, torch.cumsum(w / w.sum(), 0)


def _clustered(g, case, sites, power, lo, extent):
    centers, cumulative = _sites(g, sites, power, lo, extent)
    hi = [o + extent for o in lo]
    px, py = _around(g, case["points"], centers, cumulative, 0.02 * extent, lo, hi)
    fx, fy = _around(g, case["polygons"], centers, cumulative, 0.02 * extent, lo, hi)
    return px, py, _footprints(g, fx, fy, 15.0 * extent / 1e5)


def _degenerate(g, case):
    """Lattice stars with 1 to 5 square holes or 2 to 4 parts; 10 % of the points on vertices, 10 % on edges at dyadic
    parameters, 10 % one ulp off such a point, the rest uniform."""
    n, extent = case["polygons"], 16384.0
    parts = torch.where(_uniform(g, n) < 0.3, _randint(g, 2, 5, n), torch.ones_like(_randint(g, 0, 1, n)))
    base = torch.round(torch.stack([_uniform(g, n, 64, extent - 192), _uniform(g, n, 64, extent - 192)], 1))
    r = _randint(g, 24, 48, n).double()
    owner = torch.repeat_interleave(torch.arange(n, device=DEV), parts)
    np_ = owner.numel()
    k = torch.arange(np_, device=DEV) - (torch.cumsum(parts, 0) - parts)[owner]
    pr = r[owner]
    cx, cy = torch.round(base[owner, 0] + k * 2.5 * pr), base[owner, 1]
    holes = torch.where(k == 0, _randint(g, 1, 6, np_), torch.zeros_like(k))
    nv = _randint(g, 8, 17, np_)
    # rings: each part's outer ring, then its holes
    per_part = 1 + holes
    ring_part = torch.repeat_interleave(torch.arange(np_, device=DEV), per_part)
    which = torch.arange(ring_part.numel(), device=DEV) - (torch.cumsum(per_part, 0) - per_part)[ring_part]
    sizes = torch.where(which == 0, nv[ring_part] + 1, torch.full_like(which, 5))
    ring = torch.repeat_interleave(torch.arange(sizes.numel(), device=DEV), sizes)
    i = torch.arange(ring.numel(), device=DEV) - (torch.cumsum(sizes, 0) - sizes)[ring]
    part = ring_part[ring]
    outer = which[ring] == 0
    i = torch.where(i == sizes[ring] - 1, torch.zeros_like(i), i)  # the closing vertex is the first one again
    # one jitter per (part, vertex), so that the closing vertex repeats the first one's
    turn = _uniform(g, np_ * 16, 0.2, 0.8)[part * 16 + i.clamp(max=15)]
    jit = _uniform(g, np_ * 16, 0.75, 1.0)[part * 16 + i.clamp(max=15)]
    ang = (i + turn) * (2 * math.pi / nv[part].double())
    ox = torch.round(cx[part] + pr[part] * jit * torch.cos(ang))
    oy = torch.round(cy[part] + pr[part] * jit * torch.sin(ang))
    slot = torch.argsort(torch.rand(np_, 9, device=DEV, generator=g), 1)[part, (which[ring] - 1).clamp(min=0)]
    step, half = torch.floor(pr * 0.28)[part], torch.floor(pr * 0.12).clamp(min=2.0)[part]
    sx = torch.tensor([-1.0, -1.0, 1.0, 1.0], dtype=torch.float64, device=DEV)[i.clamp(max=3)]
    sy = torch.tensor([-1.0, 1.0, 1.0, -1.0], dtype=torch.float64, device=DEV)[i.clamp(max=3)]
    x = torch.where(outer, ox, cx[part] + (slot % 3 - 1) * step + sx * half)
    y = torch.where(outer, oy, cy[part] + (slot // 3 - 1) * step + sy * half)
    polys = _Polygons(x, y, sizes, per_part, parts)
    edge = torch.nonzero(ring[1:] == ring[:-1]).reshape(-1)  # edge e: vertices e, e + 1
    m = case["points"]
    v, e, u = m // 10, m // 10, m // 10
    at = edge[_randint(g, 0, edge.numel(), v + e + u)]
    t = _randint(g, 1, 1024, v + e + u).double() / 1024.0
    t[:v] = 0.0
    ex, ey = x[at] + t * (x[at + 1] - x[at]), y[at] + t * (y[at + 1] - y[at])
    ulp = torch.arange(v + e + u, device=DEV) >= v + e
    axis, sign = _randint(g, 0, 2, v + e + u), torch.where(_randint(g, 0, 2, v + e + u) == 1, math.inf, -math.inf).double()
    ex = torch.where(ulp & (axis == 0), torch.nextafter(ex, sign), ex)
    ey = torch.where(ulp & (axis == 1), torch.nextafter(ey, sign), ey)
    rest = m - (v + e + u)
    perm = torch.randperm(m, device=DEV, generator=g)
    px = torch.cat([_uniform(g, rest, 0, extent), ex])[perm]
    py = torch.cat([_uniform(g, rest, 0, extent), ey])[perm]
    return px, py, polys


def _data(case, seed):
    """(points' x, y, polygons) of a case."""
    g = _gen(seed)
    if case["data"] == "star":
        return _uniform(g, case["points"], 0, 1000), _uniform(g, case["points"], 0, 1000), _stars(g, case["polygons"])
    if case["data"] == "utm":  # a 100 km frame of projected coordinates, 64 equal clusters
        return _clustered(g, case, 64, 0.0, (5.0e5, 3.0e6), 1.0e5)
    if case["data"] == "zipf":  # 1024 clusters of Zipf(1.1) weights
        return _clustered(g, case, 1024, 1.1, (0.0, 0.0), 1000.0)
    return _degenerate(g, case)


def _batch_sizes(case):
    """Log-uniform job sizes, from a thousandth of the largest to the largest."""
    out = []
    for j in range(case["jobs"]):
        f = (j * 0.6180339887498949) % 1.0  # evenly spread over [0, 1)
        h = (j * 0.7548776662466927 + 0.5) % 1.0
        out.append((max(100, int(case["points"] * 1000.0 ** -f)), max(10, int(case["polygons"] * 1000.0 ** -h))))
    return out


def _wkb_points(x, y):
    n = x.numel()
    rec = torch.zeros(n, 21, dtype=torch.uint8, device=DEV)
    rec[:, 0] = 1
    rec[:, 1] = 1
    rec[:, 5:13] = x.view(torch.uint8).reshape(n, 8)
    rec[:, 13:21] = y.view(torch.uint8).reshape(n, 8)
    return rec.reshape(-1), torch.arange(n + 1, dtype=torch.int64, device=DEV) * 21


def _wkb_polygons(p):
    """Little-endian WKB of one-ring polygons: order, type, ring count, point count, coordinates."""
    ring_off = p.ring_off.long()
    m = ring_off.numel() - 1
    sizes = ring_off[1:] - ring_off[:-1]
    off = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(13 + 16 * sizes, 0, out=off[1:])
    out = torch.zeros(int(off[-1]), dtype=torch.uint8, device=DEV)
    out[off[:-1]] = 1
    out[off[:-1] + 1] = 3
    out[off[:-1] + 5] = 1
    count = sizes.to(torch.int32).contiguous().view(torch.uint8).reshape(m, 4)
    out[off[:-1, None] + 9 + torch.arange(4, device=DEV)] = count
    row = torch.repeat_interleave(torch.arange(m, device=DEV), sizes)
    at = off[row] + 13 + 16 * (torch.arange(row.numel(), device=DEV) - ring_off[row])
    byte = torch.arange(8, device=DEV)
    out[at[:, None] + byte] = p.x.view(torch.uint8).reshape(-1, 8)
    out[at[:, None] + 8 + byte] = p.y.view(torch.uint8).reshape(-1, 8)
    return out, off


def _export_inputs(case, seed):
    """Sorted unique pairs, some points with none and some with several, and attribute codes of both sides."""
    g = _gen(seed)
    n, m = case["points"], case["polygons"]
    key = torch.unique(_randint(g, 0, n, case["pairs"]) * m + _randint(g, 0, m, case["pairs"]))
    left, right = (key // m).to(torch.int32), (key % m).to(torch.int32)
    codes = (None, None)
    if case["attribute"]:
        codes = (_randint(g, 0, 7, n), _randint(g, 0, 7, m))
    return left, right, codes


# ---------------------------------------------------------------------------------------------------- prepare, run --
def _buffers(rows, count, dtype=torch.int32):
    return [torch.full((rows,), -1, dtype=dtype, device=DEV) for _ in range(count)]


def _capacity(case):
    """Pair buffers that every seed's result fits in."""
    return 8192 + int(2.0 * _pairs(case))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "export":
        left, right, codes = _export_inputs(case, seed)
        return {"kind": kind, "ctx": _abi.default_context(0), "left": left, "right": right, "codes": codes,
                "n": case["points"], "m": case["polygons"], "how": _abi.HOW_CODES[case["how"]],
                "out": _buffers(case["pairs"] + case["points"] + case["polygons"], 3, torch.int64)}
    if kind == "batch":
        return _prepare_batch(case, seed)
    px, py, polys = _data(case, seed)
    if kind == "aggregate":
        x, y, ring_off, part_off, geom_off = polys.host()
        return {"kind": kind, "points": vsb.points_from_xy(px.cpu().numpy(), py.cpu().numpy()),
                "regions": GeometryArray.from_polygon_buffers(x, y, ring_off, part_off, geom_off),
                "values": _values(case, seed).cpu().numpy(), "predicate": case["predicate"]}
    ctx = _abi.default_context(0)
    if kind == "wkb":
        return {"kind": kind, "ctx": ctx, "points": _wkb_points(px, py), "polygons": _wkb_polygons(polys)}
    state = {"kind": kind, "ctx": ctx, "keep": (px, py, polys), "points": _abi.make_points(px, py),
             "pairs": _buffers(_capacity(case), 2)}
    if kind == "build_join":
        return {**state, "polygons": polys.struct(), "predicate": PREDICATES[case["predicate"]]}
    if kind in ("nearest", "nearest_polygons"):
        state["distances"] = _buffers(_capacity(case), 1, torch.float64)[0]
    if kind == "nearest_polygons":
        return {**state, "polygons": polys.struct(), "index": _abi.point_index(ctx, px, py)}
    if kind == "join":
        state.update(predicate=PREDICATES[case["predicate"]], method=METHODS[case["method"]])
    if kind == "dwithin":
        state["distance"] = case["distance"]
    state["index"] = _abi.DeviceIndex(ctx, polys.struct(), learned=case.get("method") != "rtree")
    return state


def _prepare_batch(case, seed):
    ctx = _abi.default_context(0)
    xs, ys, keep, indexes, start = [], [], [], [], [0]
    for j, (points, polygons) in enumerate(_batch_sizes(case)):
        px, py, polys = _data({"data": "star", "points": points, "polygons": polygons}, seed * 100_003 + j + 1)
        xs.append(px)
        ys.append(py)
        keep.append(polys)
        start.append(start[-1] + points)
        indexes.append(_abi.DeviceIndex(ctx, polys.struct(), learned=True))
    x, y = torch.cat(xs), torch.cat(ys)
    plan = _abi.BatchPlan(ctx, indexes, _abi.make_points(x, y), start, options={"method": _abi.METHOD_LEARNED},
                          keepalive=(x, y, keep))
    return {"kind": "batch", "ctx": ctx, "plan": plan, "predicate": PREDICATES[case["predicate"]],
            "pairs": _buffers(_capacity(case), 2)}


def run(state):
    kind = state["kind"]
    if kind == "aggregate":
        frame = state["points"].sindex.query_aggregate(state["regions"], {"n": "size", "sum": (state["values"], "sum")},
                                                       predicate=state["predicate"])
        return frame["n"].to_numpy(), frame["sum"].to_numpy()
    if kind == "wkb":
        return [_abi.wkb_decode(state["ctx"], *state[column])[1] for column in ("points", "polygons")]
    if kind == "export":
        return _run_export(state)
    left, right = state["pairs"]
    if kind == "join":
        n, _ = state["index"].join_into(state["points"], state["predicate"], state["method"], left, right, sort=True)
        return n, left, right
    if kind == "batch":  # pairs in row order: each job's are then one run
        n, _ = state["plan"].run_into(state["predicate"], left, right)
        _abi.sort_pairs(state["ctx"], left[:n], right[:n])
        return n, left, right
    if kind == "build_join":
        index = _abi.DeviceIndex(state["ctx"], state["polygons"], learned=True)
        n, _ = index.join_into(state["points"], state["predicate"], _abi.METHOD_LEARNED, left, right, sort=True)
        index.close()
        return n, left, right
    if kind == "dwithin":
        n, _ = state["index"].dwithin_into(state["points"], left, right, distance=state["distance"], sort=True)
        return n, left, right
    if kind == "nearest":
        n, _ = state["index"].nearest_into(state["points"], left, right, state["distances"], sort=True)
        return n, left, right, state["distances"]
    n = ctypes.c_int64(0)
    stats = _abi.JoinStats()
    status = _abi.load().vs_join_nearest_polygons(
        state["ctx"].handle, state["index"].handle, ctypes.byref(state["polygons"]), math.inf, _abi.JOIN_SORT,
        left.data_ptr(), right.data_ptr(), state["distances"].data_ptr(), left.numel(), ctypes.byref(n),
        ctypes.byref(stats))
    _abi.check(status, required=n.value)
    return n.value, left, right, state["distances"]


def _run_export(state):
    n = ctypes.c_int64(0)
    codes = [None if c is None else c.data_ptr() for c in state["codes"]]
    out = state["out"]
    status = _abi.load().vs_join_export(
        state["ctx"].handle, state["left"].data_ptr(), state["right"].data_ptr(), state["left"].numel(), state["n"],
        state["m"], state["how"], *codes, *[t.data_ptr() for t in out], out[0].numel(), ctypes.byref(n))
    _abi.check(status, required=n.value)
    return n.value, out


# ------------------------------------------------------------------------------------------------ work, tolerance --
# vertices (closing one included) and rings of a polygon, and pairs for each point and polygon of the frame: means over
# seeds and sizes
_VERTICES = {"star": 37.0, "utm": 7.34, "zipf": 7.34, "degenerate": 35.9}
_RINGS = {"star": 1.0, "utm": 1.0, "zipf": 1.0, "degenerate": 4.6}
_PAIRS = {"star": 3.1e-4, "utm": 1.0e-7, "zipf": 2.4e-7, "degenerate": 1.7e-5}


def _pairs(case):
    """Pairs of a case (mean over seeds)."""
    if case["kind"] == "batch":
        return sum(n * m for n, m in _batch_sizes(case)) * _PAIRS["star"]
    points, polygons = case["points"], case["polygons"]
    pairs = points * polygons * _PAIRS[case["data"]]
    if case["data"] == "degenerate":  # the points placed on edges and vertices meet a polygon each
        pairs = 0.22 * points + (pairs if case["predicate"] != "touches" else 0.0)
    if case.get("predicate") == "bbox":  # the boxes of rotated shapes
        pairs *= 2.2
    if case["kind"] == "dwithin":  # the footprints grown by the distance
        pairs *= (1.0 + 2.0 * case["distance"] / 0.165) ** 2
    if case["kind"] == "nearest":  # at least one row each
        pairs = max(pairs, points)
    if case["kind"] == "nearest_polygons":
        pairs = max(pairs, polygons)
    return pairs


def _values(case, seed):
    return _uniform(_gen(seed + 1_000_003), case["points"], 0.0, 100.0)


def _input_bytes(data, points, polygons):
    return 16.0 * points + polygons * (16.0 * _VERTICES[data] + 4.0 * _RINGS[data] + 8.0)


def work(case):
    kind = case["kind"]
    if kind == "export":  # pairs and codes in, three 64-bit indexers out
        rows = case["pairs"] / (7 if case["attribute"] else 1)
        rows += (case["points"] if case["how"] in ("left", "outer") else 0)
        rows += (case["polygons"] if case["how"] in ("right", "outer") else 0)
        codes = 8.0 * (case["points"] + case["polygons"]) if case["attribute"] else 0.0
        return {"bytes": 8.0 * case["pairs"] + codes + 24.0 * rows}
    if kind == "batch":
        total = 0.0
        for points, polygons in _batch_sizes(case):
            total += _input_bytes("star", points, polygons)
        return {"bytes": total + 8.0 * _pairs(case)}
    data, points, polygons = case["data"], case["points"], case["polygons"]
    if kind == "wkb":  # WKB and offsets in, tags, point coordinates, offsets and polygon coordinates out
        vertices = _VERTICES[data] * polygons
        return {"bytes": points * (21.0 + 8 + 17 + 4) + polygons * (13.0 + 8 + 17 + 12) + vertices * 32.0}
    if kind == "aggregate":  # a value per point in, a count and a sum per polygon out
        return {"bytes": _input_bytes(data, points, polygons) + 8.0 * points + 16.0 * polygons}
    per_pair = 16.0 if kind in ("nearest", "nearest_polygons") else 8.0
    return {"bytes": _input_bytes(data, points, polygons) + per_pair * _pairs(case)}


def tolerance(case):
    """Pair sets, decoded columns and indexers are decided exactly, and distances follow one stated order of rounded
    operations, so every result is the same to the bit."""
    return "exact"


# ---------------------------------------------------------------------------------------------------------- exact --
_BRUTE = 2.0e10  # point-edge tests that a plain comparison of everything with everything may take


def _edges(p):
    """Start and end of every edge and its polygon (one-ring polygons)."""
    ring_off = p.ring_off.long()
    ring = torch.repeat_interleave(torch.arange(ring_off.numel() - 1, device=DEV), ring_off[1:] - ring_off[:-1])
    a = torch.nonzero(ring[1:] == ring[:-1]).reshape(-1)
    return p.x[a], p.y[a], p.x[a + 1], p.y[a + 1], ring[a]


def _brute(px, py, p, want):
    """``want(crossings odd, squared distance)`` of every (chunk of points, polygon) block, chunk by chunk."""
    ax, ay, bx, by, poly = _edges(p)
    m = p.ring_off.numel() - 1
    step = max(1, int(4.0e7 // ax.numel()))
    for i in range(0, px.numel(), step):
        x, y = px[i:i + step, None], py[i:i + step, None]
        cross = ((ay > y) != (by > y)) & (x < (bx - ax) * (y - ay) / (by - ay) + ax)
        odd = torch.zeros(x.numel(), m, dtype=torch.int32, device=DEV)
        odd.index_add_(1, poly, cross.to(torch.int32))
        dist = None
        if want == "distance":
            dx, dy = bx - ax, by - ay
            t = (((x - ax) * dx + (y - ay) * dy) / (dx * dx + dy * dy)).clamp(0.0, 1.0)
            d = (x - ax - t * dx) ** 2 + (y - ay - t * dy) ** 2
            dist = torch.full((x.numel(), m), math.inf, dtype=torch.float64, device=DEV)
            dist.scatter_reduce_(1, poly.expand(x.numel(), -1), d, "amin")
            dist = torch.where((odd & 1) == 1, torch.zeros_like(dist), dist.sqrt())
        yield i, (odd & 1) == 1, dist


def _padded(values, rows):
    out = torch.full((rows,), -1, dtype=values.dtype, device=DEV)
    out[:values.numel()] = values
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "export":
        return _exact_export(case, seed)
    if kind == "batch":
        return None
    if kind == "wkb":  # the coordinates; the rest is whole numbers
        px, py, polys = _data(case, seed)
        rest = {"tags": None, "geom_off": None, "part_off": None, "ring_off": None}
        return [{**rest, "px": px, "py": py, "x": None, "y": None},
                {**rest, "px": None, "py": None, "x": polys.x, "y": polys.y}]
    points, polygons = case["points"], case["polygons"]
    # points on the boundary need exact signs, boxes another test than the crossings
    if case["data"] == "degenerate" or case.get("predicate") in ("bbox", "touches"):
        return None
    if points * polygons * _VERTICES[case["data"]] > _BRUTE:
        return None
    px, py, polys = _data(case, seed)
    if kind == "aggregate":
        values = _values(case, seed)
        count = torch.zeros(polygons, dtype=torch.int64, device=DEV)
        total = torch.zeros(polygons, dtype=torch.float64, device=DEV)
        for i, inside, _ in _brute(px, py, polys, "inside"):
            count += inside.sum(0)
            total += (inside * values[i:i + inside.shape[0], None]).sum(0)
        return count, total
    rows, cols, far = [], [], []
    measure = "inside" if kind in ("join", "build_join") else "distance"
    if kind == "nearest_polygons":
        best = torch.full((polygons,), math.inf, dtype=torch.float64, device=DEV)
        for i, _, d in _brute(px, py, polys, measure):
            best = torch.minimum(best, d.min(0).values)
    for i, hit, d in _brute(px, py, polys, measure):
        if kind == "dwithin":
            hit = d <= case["distance"]
        elif kind == "nearest":
            hit = d == d.min(1, keepdim=True).values
        elif kind == "nearest_polygons":
            hit = d == best
        hit = torch.nonzero(hit)
        rows.append(hit[:, 0] + i)
        cols.append(hit[:, 1])
        if d is not None:
            far.append(d[hit[:, 0], hit[:, 1]])
    out = [torch.cat(t) for t in ((rows, cols, far) if far else (rows, cols))]
    if kind == "nearest_polygons":
        out = [out[1], out[0], out[2]]
        order = torch.argsort(out[0] * points + out[1])
        out = [t[order] for t in out]
    out[:2] = [t.to(torch.int32) for t in out[:2]]
    if kind not in ("nearest", "nearest_polygons"):
        out = out[:2]
    return (out[0].numel(), *(_padded(t, _capacity(case)) for t in out))


def _exact_export(case, seed):
    left, right, (left_code, right_code) = _export_inputs(case, seed)
    left, right = left.long(), right.long()
    src = torch.arange(left.numel(), device=DEV)
    if left_code is not None:
        keep = left_code[left] == right_code[right]
        left, right, src = left[keep], right[keep], src[keep]
    n, m, how = case["points"], case["polygons"], case["how"]
    minus = lambda t: torch.full_like(t, -1)  # noqa: E731
    if how in ("left", "outer"):
        alone = torch.nonzero(torch.bincount(left, minlength=n) == 0).reshape(-1)
        right_alone = torch.nonzero(torch.bincount(right, minlength=m) == 0).reshape(-1)
        left, right, src = torch.cat([left, alone]), torch.cat([right, minus(alone)]), torch.cat([src, minus(alone)])
        order = torch.sort(left, stable=True).indices
        left, right, src = left[order], right[order], src[order]
        if how == "outer":
            left, right, src = (torch.cat([left, minus(right_alone)]), torch.cat([right, right_alone]),
                                torch.cat([src, minus(right_alone)]))
    elif how == "right":
        alone = torch.nonzero(torch.bincount(right, minlength=m) == 0).reshape(-1)
        left, right, src = torch.cat([left, minus(alone)]), torch.cat([right, alone]), torch.cat([src, minus(alone)])
        order = torch.sort(right, stable=True).indices
        left, right, src = left[order], right[order], src[order]
    rows = case["pairs"] + n + m
    return left.numel(), [_padded(t, rows) for t in (left, right, src)]
