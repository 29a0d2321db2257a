"""Performance cases of the spatial-join library: what its users call, over the range they use.

A case is a dict of plain values; ``prepare`` makes its inputs from a seed on
the GPU (and, where the call takes host buffers or a file, on the host),
``run`` makes one pass through the public entry points of
``sedona_gpuspatial`` and returns everything the call returns.  Shapes and
distributions are those of the repository's five workloads
(``sedona_gpuspatial.datagen``) at the sizes of its tests and benchmark:
uniform and Gaussian-mixture points, small regular "building" polygons, large
star-shaped "zone" polygons.
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sedona-db_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from sedona_gpuspatial import capi, geoparquet, materialize  # noqa: E402
from sedona_gpuspatial.wkb import WkbColumn  # noqa: E402

EXTENT = 1e5  # side of the square the zone, building and GMM inputs live in


# ---------------------------------------------------------------------------
# the cases

def listed():
    return [
        # One DataFusion record batch through the reference's two C ABI calls (index probe, then
        # refine), host buffers in and out: the latency of the drop-in boundary.
        {"name": "abi_batch_8192_points", "kind": "abi", "rows": 8192, "build": 10_000,
         "shape": "stars", "predicate": "intersects"},
        # One record batch of building polygons through the fused join (query_batch), host
        # buffers in and out, an odd row count.
        {"name": "batch_16411_buildings", "kind": "batch", "rows": 16_411, "build": 5_000,
         "shape": "zones", "probe": "buildings", "predicate": "intersects", "large": False},
        # Point in polygon on device columns, 1M x 10k (the smallest benchmark workload).
        {"name": "pip_1m_x_10k", "kind": "join", "rows": 1_000_000, "build": 10_000,
         "shape": "stars", "probe": "uniform", "predicate": "intersects", "large": False,
         "holes": False, "nulls": False},
        # The headline join: 2M buildings x 50k zones, ST_Intersects, device columns.
        {"name": "buildings_2m_x_50k", "kind": "join", "rows": 2_000_000, "build": 50_000,
         "shape": "zones", "probe": "buildings", "predicate": "intersects", "large": False,
         "holes": False, "nulls": False},
        # Containment with holed zones, int64 offsets and null probe rows, an odd size.
        {"name": "contains_300k_holes_nulls", "kind": "join", "rows": 300_007, "build": 20_000,
         "shape": "zones", "probe": "buildings", "predicate": "contains", "large": True,
         "holes": True, "nulls": True},
        # A probe stream of uneven record batches of GPS-like points against the zones.
        {"name": "stream_4m_x_50k", "kind": "stream", "rows": 4_000_000, "build": 50_000,
         "predicate": "contains"},
        # Distance join of clustered points, 25 m.
        {"name": "dwithin_4m_x_400k", "kind": "dwithin", "rows": 4_000_000, "build": 400_000,
         "distance": 25.0},
        # Eight nearest neighbours of clustered points.
        {"name": "knn8_4m_x_400k", "kind": "knn", "rows": 4_000_000, "build": 400_000, "k": 8},
        # Small range boxes against a learned index over 20M points.
        {"name": "learned_boxes_2m_x_20m", "kind": "learned", "rows": 2_000_000,
         "build": 20_000_000, "probe": "boxes"},
        # One GeoParquet file of building polygons (Snappy) read from the page cache to the device.
        {"name": "geoparquet_400k", "kind": "geoparquet", "rows": 400_000, "shape": "buildings",
         "compression": "snappy", "version": 1, "nulls": False},
        # Output columns of one joined batch (ids, a name, the probe WKB) and the outer join's
        # unmatched rows.
        {"name": "joined_batch_4m_pairs", "kind": "materialize", "rows": 4_000_000,
         "probe_rows": 500_000, "build": 50_000, "nulls": True},
        # A query's build side: decode, bands, grids and index of 50k zones, then its first
        # record batch.
        {"name": "build_zones_50k", "kind": "build", "rows": 8192, "build": 50_000,
         "shape": "zones"},
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of [lo, hi], odd ones among them."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["abi", "batch", "join", "join", "join", "stream", "dwithin", "knn",
                       "learned", "geoparquet", "materialize", "build"])
    if kind == "abi":
        return {"kind": kind, "rows": _size(rng, 1024, 131_072), "build": _size(rng, 500, 20_000),
                "shape": "stars", "predicate": rng.choice(["intersects", "contains"])}
    if kind == "batch":
        return {"kind": kind, "rows": _size(rng, 1024, 131_072), "build": _size(rng, 500, 20_000),
                "shape": "zones", "probe": rng.choice(["gmm", "buildings"]),
                "predicate": rng.choice(["intersects", "contains", "covers"]),
                "large": rng.random() < 0.5}
    if kind == "join":
        probe = rng.choice(["uniform", "gmm", "buildings", "buildings"])
        build = _size(rng, 1000, 50_000)
        predicate = rng.choice(["intersects", "intersects", "contains", "covers"])
        # the containment tests of polygons cost about twice what intersects does
        most = 3.5e10 if probe == "buildings" and predicate != "intersects" else 7.5e10
        return {"kind": kind, "rows": min(_size(rng, 8192, 1_500_000), int(most // build)),
                "build": build, "shape": rng.choice(["stars", "zones", "zones"]), "probe": probe,
                "predicate": predicate, "large": rng.random() < 0.3, "holes": rng.random() < 0.3,
                "nulls": rng.random() < 0.3}
    if kind == "stream":
        return {"kind": kind, "rows": _size(rng, 50_000, 4_000_000),
                "build": _size(rng, 1000, 50_000), "predicate": rng.choice(["contains",
                                                                            "intersects"])}
    if kind == "dwithin":
        return {"kind": kind, "rows": _size(rng, 20_000, 4_000_000),
                "build": _size(rng, 10_000, 400_000),
                "distance": round(math.exp(rng.uniform(math.log(2.0), math.log(30.0))), 2)}
    if kind == "knn":
        return {"kind": kind, "rows": _size(rng, 10_000, 4_000_000),
                "build": _size(rng, 5_000, 400_000), "k": rng.choice([1, 2, 4, 5, 8, 10, 16])}
    if kind == "learned":
        return {"kind": kind, "rows": _size(rng, 50_000, 2_000_000),
                "build": _size(rng, 500_000, 20_000_000), "probe": rng.choice(["boxes",
                                                                               "lookups"])}
    if kind == "geoparquet":
        return {"kind": kind, "rows": _size(rng, 20_000, 400_000),
                "shape": rng.choice(["buildings", "points"]),
                "compression": rng.choice(["snappy", "none"]), "version": rng.choice([1, 2]),
                "nulls": rng.random() < 0.5}
    if kind == "materialize":
        return {"kind": kind, "rows": _size(rng, 20_000, 4_000_000),
                "probe_rows": _size(rng, 8192, 500_000), "build": _size(rng, 1000, 50_000),
                "nulls": rng.random() < 0.5}
    return {"kind": "build", "rows": 8192, "build": _size(rng, 1000, 50_000),
            "shape": rng.choice(["zones", "stars", "buildings", "points"])}


# ---------------------------------------------------------------------------
# inputs, made on the GPU

def _gen(seed, stream):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + stream)


def _u(g, n, lo, hi):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _ints(g, n, lo, hi):
    """Uniform integers in [lo, hi]."""
    return torch.randint(lo, hi + 1, (n,), generator=g, device="cuda")


def _mixture(g, components, sig_lo, sig_hi):
    return (_u(g, components, 0.0, EXTENT), _u(g, components, 0.0, EXTENT),
            _u(g, components, sig_lo, sig_hi))


def _gmm(g, n, mix):
    """n points of an equal-weight Gaussian mixture, clipped to the square."""
    mx, my, sg = mix
    c = _ints(g, n, 0, len(mx) - 1)
    z = torch.randn((2, n), generator=g, device="cuda", dtype=torch.float64)
    return ((mx[c] + sg[c] * z[0]).clamp_(0.0, EXTENT), (my[c] + sg[c] * z[1]).clamp_(0.0, EXTENT))


def _rings(nv, x, y):
    """Closes rings of nv vertices each: (points per ring, (total, 2) vertices)."""
    n = len(nv)
    start = torch.cumsum(nv, 0) - nv
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), nv)
    out = torch.empty((len(x) + n, 2), dtype=torch.float64, device="cuda")
    at = torch.arange(len(x), device="cuda") + row
    out[at, 0], out[at, 1] = x, y
    close = start + nv + torch.arange(n, device="cuda")
    out[close, 0], out[close, 1] = x[start], y[start]
    return nv + 1, out


def _stars(g, n, lo, hi, cx, cy, r_lo, r_hi):
    """Star-shaped polygons: vertices at sorted random angles, radii R * U(0.6, 1)."""
    nv = _ints(g, n, lo, hi)
    R = _u(g, n, r_lo, r_hi)
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), nv)
    turn = torch.sort(row + _u(g, len(row), 0.0, 1.0))[0] - row
    rad = R[row] * _u(g, len(row), 0.6, 1.0)
    ang = 2 * math.pi * turn
    return _rings(nv, cx[row] + rad * torch.cos(ang), cy[row] + rad * torch.sin(ang))


def _regular(g, n, cx, cy, nv=None):
    """Building-like regular polygons of 4 to 12 sides, 5 to 50 long."""
    nv = _ints(g, n, 4, 12) if nv is None else nv
    side, rot = _u(g, n, 5.0, 50.0), _u(g, n, 0.0, 2 * math.pi)
    circ = side / (2.0 * torch.sin(math.pi / nv))
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), nv)
    k = torch.arange(len(row), device="cuda") - (torch.cumsum(nv, 0) - nv)[row]
    ang = rot[row] + 2 * math.pi * k / nv[row]
    return _rings(nv, cx[row] + circ[row] * torch.cos(ang), cy[row] + circ[row] * torch.sin(ang))


def _bytes(t):
    return t.contiguous().view(torch.uint8)


def _point_wkb(x, y):
    """(row sizes, bytes) of little-endian WKB points."""
    n = len(x)
    data = torch.empty((n, 21), dtype=torch.uint8, device="cuda")
    data[:, :5] = torch.tensor([1, 1, 0, 0, 0], dtype=torch.uint8, device="cuda")
    data[:, 5:] = _bytes(torch.stack([x, y], 1))
    return torch.full((n,), 21, dtype=torch.int64, device="cuda"), data.reshape(-1)


def _polygon_wkb(npts, xy, hole=None):
    """(row sizes, bytes) of little-endian WKB polygons of one ring, or two with `hole`, whose
    rings have as many points as the outer ones."""
    n = len(npts)
    second = hole is not None
    sizes = 13 + 16 * npts + (4 + 16 * npts if second else 0)
    off = torch.cumsum(sizes, 0) - sizes
    data = torch.empty(int(sizes.sum()), dtype=torch.uint8, device="cuda")
    head = torch.zeros((n, 13), dtype=torch.uint8, device="cuda")
    head[:, 0], head[:, 1], head[:, 5] = 1, 3, 2 if second else 1
    head[:, 9:] = _bytes(npts.to(torch.int32)).view(n, 4)
    data[off[:, None] + torch.arange(13, device="cuda")] = head
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), npts)
    k = torch.arange(len(row), device="cuda") - (torch.cumsum(npts, 0) - npts)[row]
    b16 = torch.arange(16, device="cuda")
    data[(off[row] + 13 + 16 * k)[:, None] + b16] = _bytes(xy).view(-1, 16)
    if second:
        at = off + 13 + 16 * npts
        data[at[:, None] + torch.arange(4, device="cuda")] = head[:, 9:]
        data[(at[row] + 4 + 16 * k)[:, None] + b16] = _bytes(hole).view(-1, 16)
    return sizes, data


class Column:
    """A WKB column on the device, as Arrow buffers."""

    def __init__(self, sizes, data, large=False, valid=None):
        off = torch.zeros(len(sizes) + 1, dtype=torch.int64, device="cuda")
        torch.cumsum(sizes, 0, out=off[1:])
        self.n = len(sizes)
        self.offsets = off if large else off.to(torch.int32)
        self.data = data
        self.validity = None
        if valid is not None:  # LSB bitmap
            bits = torch.zeros((self.n + 7) // 8 * 8, dtype=torch.int32, device="cuda")
            bits[:self.n] = valid.to(torch.int32)
            weight = 1 << torch.arange(8, device="cuda", dtype=torch.int32)
            self.validity = (bits.view(-1, 8) * weight).sum(1).to(torch.uint8)

    def view(self):
        return capi.SpjDeviceWkb(
            length=self.n, offsets=self.offsets.data_ptr(),
            offsets_are_64bit=int(self.offsets.dtype == torch.int64), data=self.data.data_ptr(),
            data_length=self.data.numel(),
            validity=self.validity.data_ptr() if self.validity is not None else None,
            validity_offset=0)

    def host(self):
        return WkbColumn(self.offsets.cpu().numpy(), self.data.cpu().numpy(),
                         self.validity.cpu().numpy() if self.validity is not None else None)


def _polygons(g, n, shape, extent):
    if shape == "buildings":
        return _regular(g, n, *_gmm(g, n, _mixture(g, 64, 200.0, 2000.0)))
    cx, cy = _u(g, n, 0.0, extent), _u(g, n, 0.0, extent)
    if shape == "zones":
        return _stars(g, n, 32, 256, cx, cy, 500.0, 3000.0) + (cx, cy)
    return _stars(g, n, 8, 64, cx, cy, 0.5 * extent / 1000.0, 5.0 * extent / 1000.0) + (cx, cy)


def _build_column(g, case):
    """The polygons of the build side and the column made of them."""
    if case["shape"] == "points":
        x, y = _gmm(g, case["build"], _mixture(g, 128, 50.0, 500.0))
        return None, Column(*_point_wkb(x, y))
    npts, xy, *centre = _polygons(g, case["build"], case["shape"], EXTENT)
    hole = None
    if case.get("holes"):  # the ring itself, a third as large and wound the other way
        row = torch.repeat_interleave(torch.arange(len(npts), device="cuda"), npts)
        last = torch.cumsum(npts, 0)[row] - 1
        back = last - (torch.arange(len(row), device="cuda") - (last + 1 - npts[row]))
        c = torch.stack([centre[0][row], centre[1][row]], 1)
        hole = c + (xy[back] - c) / 3.0
    return (npts, xy), Column(*_polygon_wkb(npts, xy, hole), large=bool(case.get("large")))


def _probe_column(g, case):
    n, probe = case["rows"], case.get("probe", "uniform")
    valid = _u(g, n, 0.0, 1.0) >= 0.02 if case.get("nulls") else None
    if probe == "buildings":
        npts, xy = _polygons(g, n, "buildings", EXTENT)
        return Column(*_polygon_wkb(npts, xy), large=case.get("large", False), valid=valid)
    x, y = (_gmm(g, n, _mixture(g, 64, 200.0, 2000.0)) if probe == "gmm"
            else (_u(g, n, 0.0, EXTENT), _u(g, n, 0.0, EXTENT)))
    return Column(*_point_wkb(x, y), large=case.get("large", False), valid=valid)


def _rects(npts, xy):
    """Outward-rounded f32 boxes of polygons, as the caller of the index gives them."""
    n = len(npts)
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), npts)[:, None].expand(-1, 2)
    lo = torch.full((n, 2), math.inf, dtype=torch.float64, device="cuda")
    hi = torch.full((n, 2), -math.inf, dtype=torch.float64, device="cuda")
    lo.scatter_reduce_(0, row, xy, "amin")
    hi.scatter_reduce_(0, row, xy, "amax")
    lo, hi = lo.cpu().numpy().astype(np.float32), hi.cpu().numpy().astype(np.float32)
    return np.ascontiguousarray(np.concatenate(
        [np.nextafter(lo, np.float32(-np.inf)), np.nextafter(hi, np.float32(np.inf))], 1))


def _batch_sizes(seed, total):
    """Uneven record batches of 1,024 to 131,072 rows."""
    r, left, sizes = np.random.default_rng(seed), total, []
    while left > 0:
        s = min(int(math.exp(r.uniform(math.log(1024), math.log(131_072)))), left)
        sizes.append(s)
        left -= s
    return sizes


def _knn_points(case, seed):
    g = _gen(seed, 4)
    mix = _mixture(g, 128, 50.0, 500.0)
    return _gmm(g, case["build"], mix), _gmm(g, case["rows"], mix)


def _prepare_materialize(case, seed):
    """Values of the seed; the row sizes and the rows that meet are the same for all seeds, the
    build rows' order among the pairs is not."""
    g, shape = _gen(seed, 5), _gen(0, 5)
    n, nb, npr = case["rows"], case["build"], case["probe_rows"]
    x, y = _gmm(g, npr, _mixture(g, 64, 200.0, 2000.0))
    wkb = Column(*_polygon_wkb(*_regular(g, npr, x, y, _ints(shape, npr, 4, 12))))
    name_len = _ints(shape, nb, 4, 24)
    name_off = torch.zeros(nb + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(name_len, 0, out=name_off[1:])
    valid = None
    if case["nulls"]:
        valid = Column(torch.zeros(nb, dtype=torch.int64, device="cuda"), wkb.data,
                       valid=_u(g, nb, 0.0, 1.0) >= 0.05).validity
    D = materialize.DeviceColumn
    # pairs as a join returns them: probe rows ascending, a fifth of the build rows unmatched
    probe_idx = torch.sort(_ints(shape, n, 0, npr - 1))[0].to(torch.int32)
    build_idx = _ints(shape, n, 0, max(0, nb * 4 // 5 - 1)).to(torch.int32)
    build_idx = build_idx[torch.argsort(_u(g, n, 0.0, 1.0))]
    return {
        "build_cols": [D(nb, values=_ints(g, nb, 0, 1 << 40)),
                       D(nb, offsets=name_off.to(torch.int32),
                         data=_ints(g, int(name_off[-1]), 97, 122).to(torch.uint8),
                         validity=valid)],
        "probe_cols": [D(npr, values=_ints(g, npr, 0, 1 << 40)),
                       D(npr, values=_u(g, npr, 0.0, 1.0)),
                       D(npr, offsets=wkb.offsets, data=wkb.data)],
        "build_idx": build_idx, "probe_idx": probe_idx}


def _most_pairs(case):
    """Room for a join's pairs: several times what the distributions give."""
    n, nb = case["rows"], case["build"]
    if case["kind"] == "dwithin":
        return int(n * nb * 6.1e-5 * (case["distance"] / 25.0) ** 2 * 4) + 65_536
    if case["kind"] == "learned":
        return int(2 * n + (n * nb * 6e-7 if case["probe"] == "boxes" else 0)) + 65_536
    if case.get("shape") == "points":  # within 500
        return 64 * n + n * nb // 20
    reach = {"stars": 304.0, "zones": 1893.0}.get(case.get("shape", "zones"), 100.0) + 50.0
    crowd = 20.0 if case.get("shape") == "buildings" else 2.0  # clustered build rows
    return int(n * nb * 3.14 * reach ** 2 / EXTENT ** 2 * crowd) + 65_536


def prepare(case, seed):
    kind = case["kind"]
    g = _gen(seed, 1)
    s = {"kind": kind, "predicate": case.get("predicate")}
    if kind in ("abi", "batch"):  # the caller's own buffers for the pairs
        s["out"] = np.zeros((2, _most_pairs(case)), np.uint32)
    elif kind in ("join", "stream", "dwithin", "learned", "build"):
        s["out"] = torch.zeros((2, _most_pairs(case)), dtype=torch.int32, device="cuda")
    if kind == "abi":
        rings, col = _build_column(g, case)
        s["index"], s["refiner"] = capi.FloatIndex2D(), capi.Refiner()
        s["index"].push_build(_rects(*rings))
        s["index"].finish_building()
        s["refiner"].init_build_schema()
        s["refiner"].push_build(col.host())
        s["refiner"].finish_building()
        x, y = _u(g, case["rows"], 0.0, EXTENT), _u(g, case["rows"], 0.0, EXTENT)
        s["rects"] = torch.stack([x, y, x, y], 1).to(torch.float32).cpu().numpy()
        s["probe"] = Column(*_point_wkb(x, y)).host()
    elif kind in ("batch", "join"):
        s["join"] = capi.SpatialJoin()
        s["build"] = _build_column(g, case)[1]
        torch.cuda.synchronize()
        s["join"].build_device(s["build"].view())
        s["probe"] = _probe_column(g, case)
        if kind == "batch":
            s["probe"] = s["probe"].host()
    elif kind == "stream":
        s["join"] = capi.SpatialJoin()
        s["build"] = _build_column(g, dict(case, shape="zones"))[1]
        torch.cuda.synchronize()
        s["join"].build_device(s["build"].view())
        x, y = _gmm(g, case["rows"], _mixture(g, 64, 200.0, 2000.0))
        s["cols"], at = [], 0
        for n in _batch_sizes(seed, case["rows"]):
            s["cols"].append(Column(*_point_wkb(x[at:at + n], y[at:at + n])))
            at += n
        torch.cuda.synchronize()
        s["stream"] = capi.StreamProbe(s["join"])
        s["stream"].set_batches([c.view() for c in s["cols"]])
    elif kind == "dwithin":
        (bx, by), (px, py) = _knn_points(case, seed)
        s["join"], s["distance"] = capi.SpatialJoin(), case["distance"]
        s["build"] = Column(*_point_wkb(bx, by))
        torch.cuda.synchronize()
        s["join"].build_device(s["build"].view())
        s["probe"] = Column(*_point_wkb(px, py))
    elif kind == "knn":
        (bx, by), (px, py) = _knn_points(case, seed)
        s["knn"], s["k"], s["n"] = capi.KnnJoin(), case["k"], case["rows"]
        s["knn"].build(bx.cpu().numpy(), by.cpu().numpy())
        s["xy"] = torch.stack([px, py], 1).contiguous()
    elif kind == "learned":
        mix = _mixture(g, 256, 50.0, 500.0)
        bx, by = _gmm(g, case["build"], mix)
        s["learned"] = capi.LearnedIndex()
        s["build"] = Column(*_point_wkb(bx, by))
        torch.cuda.synchronize()
        s["learned"].build_device(s["build"].view())
        if case["probe"] == "boxes":
            cx, cy = _gmm(g, case["rows"], mix)
            h = torch.exp(_u(g, case["rows"], math.log(0.01), math.log(10.0))) / 2
            ring = torch.stack([torch.stack([cx - h, cy - h], 1), torch.stack([cx + h, cy - h], 1),
                                torch.stack([cx + h, cy + h], 1), torch.stack([cx - h, cy + h], 1),
                                torch.stack([cx - h, cy - h], 1)], 1).reshape(-1, 2)
            s["probe"] = Column(*_polygon_wkb(
                torch.full((case["rows"],), 5, dtype=torch.int64, device="cuda"), ring))
        else:
            pick = _ints(g, case["rows"], 0, case["build"] - 1)
            s["probe"] = Column(*_point_wkb(bx[pick], by[pick]))
    elif kind == "geoparquet":
        shape = _gen(0, 9)  # row sizes and nulls are the file's, its coordinates the seed's
        valid = _u(shape, case["rows"], 0.0, 1.0) >= 0.02 if case["nulls"] else None
        x, y = _gmm(g, case["rows"], _mixture(g, 64, 200.0, 2000.0))
        if case["shape"] == "points":
            sizes, data = _point_wkb(x, y)
        else:
            sizes, data = _polygon_wkb(*_regular(g, case["rows"], x, y,
                                                 _ints(shape, case["rows"], 4, 12)))
        s["dir"] = tempfile.TemporaryDirectory(prefix="spj_cases_")
        s["path"] = os.path.join(s["dir"].name, "column.parquet")
        geoparquet.write_wkb(s["path"], Column(sizes, data, valid=valid).host(),
                             compression=case["compression"], page_version=case["version"])
    elif kind == "materialize":
        s.update(_prepare_materialize(case, seed))
    elif kind == "build":
        s["build"] = _build_column(g, case)[1]
        s["probe"] = _probe_column(g, dict(case, probe="gmm"))
        # a build side of points serves a distance join
        s["predicate"], s["distance"] = (("dwithin", 500.0) if case["shape"] == "points"
                                         else ("intersects", 0.0))
    else:
        raise ValueError(kind)
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# one pass

class _Device:
    """A result buffer of the library; `owner` (a join, an open file) lives as long as its tensors."""

    def __init__(self, ptr, n, kind, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": kind, "data": (ptr, False),
                                         "version": 3, "strides": None}


def _on_device(owner, ptr, n, kind="<i4"):
    """A tensor over the library's own result buffer."""
    if not n:
        return torch.empty(0, dtype={"<i4": torch.int32, "<i8": torch.int64}.get(kind, torch.uint8),
                           device="cuda")
    return torch.as_tensor(_Device(ptr, n, kind, owner), device="cuda")


def _keep(state, source, pairs):
    """The pairs in the caller's buffers, copied on the stream of the join that owns them."""
    db, dp, n = pairs
    out = state["out"]
    with torch.cuda.stream(torch.cuda.ExternalStream(source.stream())):
        out[0, :n].copy_(_on_device(None, db, n))
        out[1, :n].copy_(_on_device(None, dp, n))
    return {"build": out[0], "probe": out[1], "count": n}


def _keep_host(state, b, p):
    out = state["out"]
    out[0, :len(b)], out[1, :len(p)] = b, p
    return {"build": out[0], "probe": out[1], "count": len(b)}


def run(state):
    kind = state["kind"]
    if kind == "abi":
        b, p = state["index"].probe(state["rects"])
        return _keep_host(state, *state["refiner"].refine(state["probe"], state["predicate"], b, p))
    if kind == "batch":
        return _keep_host(state, *state["join"].probe(state["probe"], state["predicate"]))
    if kind == "join":
        join = state["join"]
        return _keep(state, join, join.probe_device(state["probe"].view(), state["predicate"]))
    if kind == "stream":
        return _keep(state, state["stream"], state["stream"].run(state["predicate"]))
    if kind == "dwithin":
        join = state["join"]
        return _keep(state, join, join.probe_device(state["probe"].view(), "dwithin",
                                                    state["distance"]))
    if kind == "knn":
        idx = torch.empty((state["n"], state["k"]), dtype=torch.int32, device="cuda")
        dist = torch.empty((state["n"], state["k"]), dtype=torch.float64, device="cuda")
        state["knn"].query_device(state["xy"].data_ptr(), state["n"], state["k"], idx.data_ptr(),
                                  dist.data_ptr())
        return {"idx": idx, "dist": dist}
    if kind == "learned":
        index = state["learned"]
        return _keep(state, index, index.query_device(state["probe"].view(), "intersects"))
    if kind == "geoparquet":
        f = geoparquet.GeoParquetFile(state["path"])  # closed with the last of its tensors
        d = f.read_wkb()
        out = {"offsets": _on_device(f, d.offsets, d.length + 1, "<i8"),
               "data": _on_device(f, d.data, d.data_length, "|u1")}
        if d.validity:
            out["validity"] = _on_device(f, d.validity, (d.length + 7) // 8, "|u1")
        return out
    if kind == "materialize":
        cols = materialize.build_joined_columns(state["build_cols"], state["probe_cols"],
                                                state["build_idx"], state["probe_idx"])
        seen = materialize.VisitedBitmap(state["build_cols"][0].length)
        seen.mark(state["build_idx"])
        out = {"unmatched": seen.collect(False)}
        for i, c in enumerate(cols):
            for part in ("values", "offsets", "data", "validity"):
                if getattr(c, part) is not None:
                    out["%d_%s" % (i, part)] = getattr(c, part)
        return out
    join = capi.SpatialJoin()  # build: a query's own join
    join.build_device(state["build"].view())
    return _keep(state, join, join.probe_device(state["probe"].view(), state["predicate"],
                                                state["distance"]))


# ---------------------------------------------------------------------------
# what a pass cannot do without

# mean sizes of the inputs: vertices per ring (closed), and the share of the square that one
# polygon covers (star area: pi R^2 times the mean of two neighbouring radii's product)
_VERTS = {"stars": 37.0, "zones": 145.0, "buildings": 9.0}
_COVER = {"stars": 3.14 * 9.25 * 0.64 / 1e6, "zones": 3.14 * 3.58e6 * 0.64 / EXTENT ** 2}


def _wkb_bytes(case, n, shape):
    off = 8 if case.get("large") else 4
    per = 21 if shape not in _VERTS else 13 + 16 * _VERTS[shape]
    if case.get("holes") and shape in ("stars", "zones"):
        per = 2 * per - 9
    return n * (per + off)


def work(case):
    """Each input byte read once, each output byte written once; operations: one segment test
    (10) per pair of a polygon join, one distance (5) per pair of a distance join or KNN."""
    kind, n, nb = case["kind"], case.get("rows", 0), case.get("build", 0)
    if kind in ("abi", "batch", "join", "stream"):
        shape = case.get("shape", "zones")
        pairs = n * nb * _COVER[shape]
        probe = _wkb_bytes(case, n, case.get("probe", "points"))
        build = nb * (16 * _VERTS[shape] + 16)  # vertices and box
        return {"bytes": probe + build + 8 * pairs, "flops": 10 * pairs}
    if kind == "dwithin":
        # neighbours of a point in the mixture, for the square's 128 clusters
        pairs = n * nb * 6.1e-5 * (case["distance"] / 25.0) ** 2
        return {"bytes": 25 * n + 16 * nb + 8 * pairs, "flops": 5 * pairs}
    if kind == "knn":
        return {"bytes": 16 * n + 16 * nb + 12 * n * case["k"], "flops": 5 * n * case["k"]}
    if kind == "learned":
        pairs = n * (nb * 1.0e-7 if case["probe"] == "boxes" else 1.0)
        per = 13 + 80 + 4 if case["probe"] == "boxes" else 25
        return {"bytes": n * per + 8 * pairs, "flops": 4 * pairs}
    if kind == "geoparquet":
        value = 21 if case["shape"] == "points" else 13 + 16 * _VERTS["buildings"]
        return {"bytes": n * (2 * value + 4 + 8), "flops": 0}
    if kind == "materialize":
        # pair ids, two ids, a double, a name of 14 bytes, a WKB value
        per = 8 + 2 * 16 + 16 + 2 * 14 + 12 + 2 * (13 + 16 * _VERTS["buildings"]) + 12
        return {"bytes": n * per + case["build"] / 4, "flops": 0}
    # build: the column read once, its vertices (f64 and f32) and boxes written once
    verts = _VERTS.get(case["shape"], 1.0)
    return {"bytes": _wkb_bytes(case, nb, case["shape"]) + nb * (24 * verts + 16),
            "flops": 10 * nb * verts}


# ---------------------------------------------------------------------------
# the same results in plain 64-bit arithmetic

def exact(case, seed):
    """KNN distances (the other outputs are whole numbers and bytes).  Probes are taken in x
    order; a chunk's k-th distance within a few thousand x neighbours bounds the x window that
    holds every probe's k nearest."""
    if case["kind"] != "knn" or case["rows"] * case["build"] > 2e12:
        return None
    (bx, by), (px, py) = _knn_points(case, seed)
    k, nb = case["k"], len(bx)
    bx, order = torch.sort(bx)
    by = by[order]
    rows = torch.argsort(px)
    out = torch.empty((len(px), k), dtype=torch.float64, device="cuda")

    def nearest(r, lo, hi):
        d2 = (px[r, None] - bx[lo:hi]).square_() + (py[r, None] - by[lo:hi]).square_()
        return torch.topk(d2, min(k, hi - lo), dim=1, largest=False)[0].sqrt()

    for r in torch.split(rows, 8192):
        x0, x1 = px[r[0]], px[r[-1]]
        mid = int(torch.searchsorted(bx, (x0 + x1) / 2))
        lo, hi = max(0, mid - 2048), min(nb, mid + 2048)
        far = nearest(r, lo, hi)[:, -1].max() if hi - lo >= k else math.inf
        lo = int(torch.searchsorted(bx, (x0 - far).reshape(1)))
        hi = int(torch.searchsorted(bx, (x1 + far).reshape(1), right=True))
        for part in torch.split(r, max(1, int(2e8) // max(1, hi - lo))):
            out[part] = nearest(part, lo, hi)
    return {"idx": None, "dist": out}
