"""The packet refine (probe rows in Morton order, 32 to a traversal) against the
candidate pairs' path and the oracle."""
import numpy as np
import pytest

from gpu_util import device_column, device_pairs, pairs

pytestmark = pytest.mark.gpu

PREDS = ["intersects", "contains", "covers", "within", "coveredby", "touches", "equals", "disjoint"]


@pytest.fixture(scope="module")
def capi():
    from sedona_gpuspatial import _build, capi
    _build.build()
    return capi


def _star(rng, c, n, r):
    ang = np.sort(rng.uniform(0, 2 * np.pi, n))
    rad = r * rng.uniform(0.6, 1.0, n)
    ring = c + np.stack([rad * np.cos(ang), rad * np.sin(ang)], 1)
    return np.vstack([ring, ring[:1]])


def _zones(rng, n, holes):
    """Stars of 5 to 120 points (with and without cell grids), some with a star
    hole, some multipolygons."""
    from sedona_gpuspatial import wkb
    out = []
    for _ in range(n):
        c = rng.uniform(0, 200, 2)
        shell = _star(rng, c, int(rng.integers(5, 120)), rng.uniform(5, 40))
        rings = [shell]
        if holes and rng.random() < 0.5:
            rings.append((c + (shell - c) / 3.0)[::-1])
        if holes and rng.random() < 0.15:
            out.append(wkb.wkb_multipolygon([rings, [_star(rng, rng.uniform(0, 200, 2), 30, 10.0)]]))
        else:
            out.append(wkb.wkb_polygon(rings))
    return out


def _probes(rng, n, kind, build):
    """Points or polygons; some rows null or empty, some on a zone's vertices."""
    from sedona_gpuspatial import wkb
    out = []
    for i in range(n):
        u = rng.random()
        if u < 0.03:
            out.append(None)
        elif u < 0.05:
            out.append(wkb.wkb_point(np.nan, np.nan))
        elif kind == "points":
            out.append(wkb.wkb_point(*rng.uniform(-5, 205, 2)))
        elif kind == "lattice":
            out.append(wkb.wkb_point(*rng.integers(0, 200, 2).astype(float)))
        elif kind == "mixed" and u < 0.3:
            out.append(wkb.wkb_point(*rng.uniform(0, 200, 2)))
        elif kind == "mixed" and u < 0.4:
            out.append(build[int(rng.integers(0, len(build)))])
        elif kind == "mixed" and u < 0.6:
            a = _star(rng, rng.uniform(0, 200, 2), 6, 6.0)
            out.append(wkb.wkb_multipolygon([[a], [_star(rng, rng.uniform(0, 200, 2), 5, 3.0)]]))
        else:
            c = rng.uniform(0, 200, 2)
            a = _star(rng, c, int(rng.integers(3, 20)), np.exp(rng.uniform(-3, 4)))
            rings = [a]
            if kind == "mixed" and u < 0.7:
                rings.append((c + (a - c) / 2.0)[::-1])
            out.append(wkb.wkb_polygon(rings))
    return out


def _both(capi, build, probe, preds):
    fast, general = capi.SpatialJoin(probe_order=1), capi.SpatialJoin(probe_order=1)
    general.set_option("candidate_order", 0)  # (any set order takes the candidate pairs' path)
    for j in (fast, general):
        j.build(build)
    for pred in preds:
        b, p = fast.probe(probe, pred)
        gb, gp = general.probe(probe, pred)
        np.testing.assert_array_equal(b, gb, err_msg=pred)
        np.testing.assert_array_equal(p, gp, err_msg=pred)
        yield pred, b, p


@pytest.mark.parametrize("kind", ["points", "lattice", "polygons", "mixed"])
@pytest.mark.parametrize("n", [2, 31, 32, 33, 127, 2500])
def test_packet_same_pairs_and_positions(capi, oracle_lib, kind, n):
    from sedona_gpuspatial import wkb
    rng = np.random.default_rng(n * 7 + len(kind))
    zones = _zones(rng, 60, holes=True)
    build = wkb.column_from_values(zones)
    if kind == "lattice":  # zones on integer vertices: points on edges and corners
        build = wkb.column_from_values([
            wkb.wkb_polygon([np.round(_star(rng, rng.integers(0, 200, 2), 40, 30.0))])
            for _ in range(60)])
    probe = wkb.column_from_values(_probes(rng, n, kind, zones))
    for pred, b, p in _both(capi, build, probe, PREDS):
        if pred != "disjoint" and n <= 127:
            ob, op = oracle_lib.join(oracle_lib.Geoms(build), oracle_lib.Geoms(probe), pred,
                                     nthreads=4)
            assert pairs(b, p) == sorted(zip(op.tolist(), ob.tolist())), pred


def test_packet_far_offset_and_huge_probes(capi):
    """Coordinates whose FP32 copies carry few digits (the undecided sides go
    to FP64 and to the full tests), and probes larger than the zones."""
    from sedona_gpuspatial import wkb
    rng = np.random.default_rng(3)
    off = np.array([4.0e6, -7.0e6])
    build = wkb.column_from_values([wkb.wkb_polygon([off + _star(rng, rng.uniform(0, 200, 2), 60, 30.0)])
                                    for _ in range(40)])
    probe = wkb.column_from_values(
        [wkb.wkb_polygon([off + _star(rng, rng.uniform(0, 200, 2), 8, np.exp(rng.uniform(-2, 6)))])
         for _ in range(1500)] +
        [wkb.wkb_point(*(off + rng.uniform(0, 200, 2))) for _ in range(500)])
    for _ in _both(capi, build, probe, PREDS):
        pass


@pytest.mark.parametrize("sizes", [(1023, 1024), (1024, 1025), (5000, 300), (65535, 65536, 70000, 40)])
def test_packet_large_rings(capi, oracle_lib, sizes):
    """Rings of both sides of what one block indexes (1,024 edges) and of what has
    an index at all (65,535), beside small ones; one whose edges crowd in a cell
    (over 255, so the grid does not answer there); with and without holes."""
    from sedona_gpuspatial import wkb
    rng = np.random.default_rng(len(sizes) + sizes[0])
    zones = []
    for k, n in enumerate(sizes):
        c = rng.uniform(60, 140, 2)
        shell = _star(rng, c, n, 60.0)
        zones.append(wkb.wkb_polygon([shell] + ([(c + (shell - c) / 3.0)[::-1]] if k % 2 else [])))
    ang = np.sort(rng.uniform(0, 2 * np.pi, 900))
    rad = np.where(np.arange(900) % 2, 40.0, 1e-3)
    spikes = 100.0 + np.stack([rad * np.cos(ang), rad * np.sin(ang)], 1)
    zones.append(wkb.wkb_polygon([np.vstack([spikes, spikes[:1]])]))
    zones += _zones(rng, 20, holes=True)
    build = wkb.column_from_values(zones)
    assert max(len(z) for z in zones) > 16 * max(sizes)
    for kind, n in (("points", 400), ("polygons", 120)):
        rows = _probes(rng, n, kind, zones)
        rows += [wkb.wkb_point(*(100.0 + rng.uniform(-0.1, 0.1, 2))) if kind == "points" else
                 wkb.wkb_polygon([_star(rng, 100.0 + rng.uniform(-2, 2, 2), 5, 1.0)])
                 for _ in range(40)]
        probe = wkb.column_from_values(rows)
        for pred, b, p in _both(capi, build, probe, PREDS):
            if pred in ("intersects", "contains"):
                ob, op = oracle_lib.join(oracle_lib.Geoms(build), oracle_lib.Geoms(probe), pred,
                                         nthreads=8)
                assert pairs(b, p) == sorted(zip(op.tolist(), ob.tolist())), pred


def test_packet_capacities_grow(capi):
    """More records and more open pairs than the first guess has room for."""
    from sedona_gpuspatial import wkb
    rng = np.random.default_rng(4)
    build = wkb.column_from_values([wkb.wkb_polygon([_star(rng, np.zeros(2), 4, 50.0)])
                                    for _ in range(40000)])
    points = wkb.column_from_values([wkb.wkb_point(*rng.uniform(-40, 40, 2)) for _ in range(40)])
    for _ in _both(capi, build, points, ["intersects"]):
        pass
    multi = wkb.column_from_values([
        wkb.wkb_multipolygon([[_star(rng, rng.uniform(-40, 40, 2), 5, 3.0)],
                              [_star(rng, rng.uniform(-40, 40, 2), 5, 3.0)]]) for _ in range(40)])
    for _ in _both(capi, build, multi, ["intersects", "contains"]):
        pass


@pytest.mark.parametrize("size", [256, 256 * 300, 0])
def test_packet_memory_limit(capi, size):
    """Records and open pairs past packet_bytes: the candidate pairs (ST_DWithin:
    the traversal per probe) answer, and the packets again with more room."""
    from sedona_gpuspatial import wkb
    rng = np.random.default_rng(11)
    zones = _zones(rng, 400, holes=True)
    build = wkb.column_from_values(zones)
    for kind in ("points", "mixed"):
        probe = wkb.column_from_values(_probes(rng, 600, kind, zones))
        j = capi.SpatialJoin(probe_order=1)
        j.build(build)
        for pred in ("intersects", "contains"):
            exp = j.probe(probe, pred)
            for limit in (size, 1 << 34):
                j.set_option("packet_bytes", limit)
                k = capi.SpatialJoin(probe_order=1)
                k.set_option("packet_bytes", limit)
                k.build(build)
                for got in (j.probe(probe, pred), k.probe(probe, pred)):
                    np.testing.assert_array_equal(exp[0], got[0])
                    np.testing.assert_array_equal(exp[1], got[1])
    bp, pp = (wkb.points_column(*rng.uniform(0, 50, (2, m))) for m in (2000, 500))
    got = []
    for limit in (1 << 34, size):
        j = capi.SpatialJoin(probe_order=1)
        j.set_option("packet_bytes", limit)
        j.build(bp)
        got.append(j.probe(pp, "dwithin", distance=4.0))
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("limit", [1 << 34, 256 * 1500])
def test_packet_stream_grows(capi, limit):
    """A stream whose records and pairs both outgrow their first room (the graph
    is captured again; only the pairs are written again), or pass the limit (the
    candidate pairs): the arrays of the unordered graph, run after run and for
    smaller batches afterwards."""
    import torch
    from sedona_gpuspatial import wkb
    rng = np.random.default_rng(12)
    build = wkb.column_from_values([wkb.wkb_polygon([_star(rng, np.zeros(2), 12, 50.0)])
                                    for _ in range(2000)])
    sizes = (900, 1, 1600, 0, 499)
    cols = [wkb.points_column(*rng.uniform(-45, 45, (2, m))) for m in sizes]
    out = []
    for order in (-1, 1):
        j = capi.SpatialJoin(probe_order=order)
        j.set_option("packet_bytes", limit)
        j.build(build)
        st = capi.StreamProbe(j)
        res = []
        for some in (cols, cols[:2], cols):
            dev = [device_column(capi, c) for c in some]
            torch.cuda.synchronize()
            st.set_batches([d for d, _ in dev])
            for pred in ("intersects", "contains", "contains"):
                db, dp, n = st.run(pred)
                res.append(device_pairs(db, dp, n))
        out.append(res)
    assert len(out[0][0][0]) > 4 * sum(sizes) + 1024
    for a, b in zip(*out):
        np.testing.assert_array_equal(a[0], b[0])
        np.testing.assert_array_equal(a[1], b[1])


@pytest.mark.parametrize("n,order,packets,launches", [
    (3000, -1, True, 10), (3000, 1, True, 10), (3000, 1, False, 16),
    (70000, -1, True, 12), (70000, 0, True, 23), (70000, 0, False, 31)])
def test_stream_launches(capi, n, order, packets, launches):
    """Launches per replay: scans and sorts of up to 16,384 elements are one each
    (the scans within the sort of 70,000 rows are of 35 tiles' 256 counts)."""
    import torch
    from sedona_gpuspatial import wkb
    rng = np.random.default_rng(13)
    j = capi.SpatialJoin(probe_order=order)
    if not packets:
        j.set_option("packet_bytes", 0)
    j.build(wkb.column_from_values(_zones(rng, 20, holes=False)))
    dev = device_column(capi, wkb.points_column(*rng.uniform(0, 200, (2, n))))
    torch.cuda.synchronize()
    st = capi.StreamProbe(j)
    st.set_batches([dev[0]])
    st.run("contains")
    assert st.stats()["launches_per_replay"] == launches


@pytest.mark.parametrize("n,leaf", [(2, 16), (31, 1), (32, 16), (33, 64), (127, 33), (2500, 16)])
def test_packet_dwithin_same_pairs_and_positions(capi, n, leaf):
    """ST_DWithin of points by the packet traversal against the traversal per
    probe: pairs exactly at d, rows with no box, points and distances outside
    the FP32 test's range, more records than the first guess holds."""
    from sedona_gpuspatial import wkb
    rng = np.random.default_rng(n)

    def points(m):
        xy = np.concatenate([rng.integers(0, 40, (m // 2, 2)).astype(np.float64),
                             rng.normal(20, 8, (m - m // 2, 2))])
        vals = [wkb.wkb_point(*v) for v in xy]
        for i, v in enumerate([None, wkb.wkb_point(1e30, 3.0), wkb.wkb_point(np.nan, np.nan),
                               wkb.wkb_point(1e-40, -1e-40)]):
            if m > 30:
                vals[i * 7] = v
        return vals

    near = [wkb.wkb_point(*v) for v in rng.integers(0, 40, (3000, 2)).astype(np.float64)]
    for vals in (near, points(3000)):  # (without and with the exact test for every pair)
        build, probe = wkb.column_from_values(vals), wkb.column_from_values(points(n))
        js = [capi.SpatialJoin(probe_order=1, leaf_size=leaf) for _ in range(2)]
        js[1].set_option("dwithin_arena", 0)  # (any set arena takes the traversal per probe)
        for j in js:
            j.build(build)
        rows = rng.choice([0.0, 1.0, 5.0, 100.0, np.inf, np.nan, -1.0, 1e-30], n)
        for d in (0.0, 5.0, np.nextafter(5.0, 0), 1e-40, 60.0, 1e200, np.inf, rows):
            got = []
            for j in js:
                if d is rows:
                    j.set_probe_distances(rows)
                got.append(j.probe(probe, "dwithin", distance=0.0 if d is rows else d))
            np.testing.assert_array_equal(got[0][0], got[1][0])
            np.testing.assert_array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("leaf", [1, 16, 33, 64])
def test_packet_dwithin_counts_the_same_candidates(capi, leaf):
    """The statistics of the packet traversal are those of the traversal per probe:
    boxes that overlap, of leaves that are not farther as a whole."""
    from sedona_gpuspatial import wkb
    rng = np.random.default_rng(leaf)
    build = wkb.points_column(*np.concatenate([rng.normal(50, 3, (2, 3000)),
                                               rng.uniform(0, 100, (2, 2000))], 1))
    probe = wkb.points_column(*rng.uniform(0, 100, (2, 700)))
    far = wkb.column_from_values([wkb.wkb_point(1e30, 1.0), wkb.wkb_point(50.0, 50.0)] * 40)
    for pts in (probe, far):
        for d in (0.0, 0.7, 6.0, 90.0):
            got = []
            for limit in (1 << 34, 0):
                j = capi.SpatialJoin(probe_order=1, leaf_size=leaf)
                j.set_option("packet_bytes", limit)
                j.build(build)
                b, _ = j.probe(pts, "dwithin", distance=d)
                st = j.stats()
                got.append((len(b), st["candidates"], st["pairs_evaluated"]))
                assert j.packet_calls() == (1 if limit else 0)
            assert got[0] == got[1]


@pytest.mark.parametrize("n", [1, 31, 4096, 4097, 8193, 16384, 16385, 20001])
@pytest.mark.parametrize("order", [-1, 1])
def test_scans_and_sorts_at_the_sizes_of_one_block(capi, n, order):
    """Build and probe rows of both sides of the sizes that one block scans and
    sorts: row i of a shuffled grid of squares meets the point of its centre."""
    from sedona_gpuspatial import wkb
    rng = np.random.default_rng(n)
    at = rng.permutation(n)
    x, y = (at % 150) * 3.0, (at // 150) * 3.0
    build = wkb.column_from_values([
        wkb.wkb_polygon([np.array([(a, b), (a + 1, b), (a + 1, b + 1), (a, b + 1), (a, b)])])
        for a, b in zip(x, y)])
    to = rng.permutation(n)
    probe = wkb.points_column(x[to] + 0.5, y[to] + 0.5)
    j = capi.SpatialJoin(probe_order=order)
    j.build(build)
    b, p = j.probe(probe, "intersects")
    np.testing.assert_array_equal(p, np.arange(n))
    np.testing.assert_array_equal(b, to)


@pytest.mark.parametrize("pred,n", [("dwithin", 2047), ("dwithin", 2048), ("contains", 8191),
                                    ("contains", 8192), ("touches", 8192)])
def test_packet_from_the_first_row_counts(capi, pred, n):
    """The sizes from which the packets are taken, against the candidate pairs."""
    from sedona_gpuspatial import wkb
    rng = np.random.default_rng(n)
    if pred == "dwithin":
        build, probe = (wkb.points_column(*rng.uniform(0, 200, (2, m))) for m in (3000, n))
    else:
        zones = _zones(rng, 60, holes=True)
        build = wkb.column_from_values(zones)
        probe = wkb.column_from_values(_probes(rng, n, "polygons", zones))
    got = []
    for option in (None, "candidate_order", "dwithin_arena"):
        j = capi.SpatialJoin()
        if option:
            j.set_option(option, 0)
        j.build(build)
        got.append(j.probe(probe, pred, distance=4.0))
    for other in got[1:]:
        np.testing.assert_array_equal(got[0][0], other[0])
        np.testing.assert_array_equal(got[0][1], other[1])
    assert len(got[0][0]) > 0 or pred == "touches"


@pytest.mark.parametrize("build_rows,radius,n,pred,distance,packets", [
    (2000, 20.0, 70000, "intersects", 0.0, 1),   # many probes in each build row's box
    (2000, 20.0, 65535, "intersects", 0.0, 0),
    (20000, 0.02, 70000, "contains", 0.0, 0),    # build rows that hardly any probe meets
    (300000, 0.0, 5000, "dwithin", 0.01, 0),     # few probes, far apart
    (300000, 0.0, 5000, "dwithin", 1.0, 1),      # many neighbours each
    (300000, 0.0, 4000, "dwithin", 0.01, 1),
    (300000, 0.0, 26000, "dwithin", 0.01, 1),
    (5000, 0.0, 20000, "dwithin", 0.01, 0)])
def test_packets_by_density(capi, build_rows, radius, n, pred, distance, packets):
    """The path that the sizes choose, with the pairs of the other one."""
    from sedona_gpuspatial import wkb
    rng = np.random.default_rng(build_rows + n)
    if radius:
        turn = np.linspace(0, 2 * np.pi, 9)
        ring = radius * np.stack([np.cos(turn), np.sin(turn)], 1)
        ring[-1] = ring[0]
        build = wkb.column_from_values([wkb.wkb_polygon([ring + c])
                                        for c in rng.uniform(0, 200, (build_rows, 2))])
    else:
        build = wkb.points_column(*rng.uniform(0, 200, (2, build_rows)))
    probe = wkb.points_column(*rng.uniform(0, 200, (2, n)))
    got = []
    for limit in (1 << 34, 0):
        j = capi.SpatialJoin()
        j.set_option("packet_bytes", limit)
        j.build(build)
        got.append(j.probe(probe, pred, distance=distance))
        assert j.packet_calls() == (packets if limit else 0)
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])
