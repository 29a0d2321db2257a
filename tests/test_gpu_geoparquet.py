"""GeoParquet read onto the device (SpjParquetReadWkb) against the values
pyarrow wrote into the committed fixtures, against the writer's input on
round trips, and through a join against the same columns given directly.
Byte data: results must match exactly."""
import os

import numpy as np
import pytest

import gpu_util

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
FIXDIR = os.path.join(HERE, "golden", "parquet")
FIXTURES = sorted(f[:-8] for f in os.listdir(FIXDIR) if f.endswith(".parquet"))


@pytest.fixture(scope="module")
def gp():
    from sedona_gpuspatial import _build
    _build.build()
    from sedona_gpuspatial import geoparquet
    return geoparquet


def _expected(name):
    z = np.load(os.path.join(HERE, "golden", "parquet_expected.npz"))
    return z[f"off_{name}"], z[f"data_{name}"], z[f"valid_{name}"]


def _assert_column(got, off, data, valid):
    """got: a host WkbColumn with int64 offsets; nulls are empty values."""
    n = len(valid)
    assert len(got) == n
    lens = np.diff(off)
    exp_off = np.zeros(n + 1, np.int64)
    exp_off[1:] = np.cumsum(np.where(valid, lens, 0))
    assert np.array_equal(got.offsets, exp_off)
    assert np.array_equal(got.data, data)
    if valid.all():
        assert got.validity is None
    else:
        bits = np.unpackbits(got.validity, bitorder="little")[:n].astype(bool)
        assert np.array_equal(bits, valid)


@pytest.mark.parametrize("name", FIXTURES)
def test_fixture_read_matches_pyarrow_values(gp, name):
    off, data, valid = _expected(name)
    with gp.GeoParquetFile(os.path.join(FIXDIR, name + ".parquet")) as f:
        for _ in range(2):  # a second read reuses the handle's buffers
            d = f.read_wkb()
            _assert_column(gp.device_to_host(d), off, data, valid)
        st = f.stats()
        assert st["value_bytes"] == len(data) and st["ms_device"] > 0


@pytest.mark.parametrize("name", ["dict_snappy_v1", "plain_snappy_v2"])
def test_row_group_ranges(gp, name):
    off, data, valid = _expected(name)
    with gp.GeoParquetFile(os.path.join(FIXDIR, name + ".parquet")) as f:
        nrg = f.info()["num_row_groups"]
        r0 = 0
        for g in range(nrg):
            rows = f.row_group_rows(g)
            d = f.read_wkb(rg_begin=g, rg_end=g + 1)
            sub_off = off[r0:r0 + rows + 1]
            _assert_column(gp.device_to_host(d), sub_off - sub_off[0],
                           data[sub_off[0]:sub_off[-1]], valid[r0:r0 + rows])
            r0 += rows
        d = f.read_wkb(rg_begin=1, rg_end=1)
        assert d.length == 0


@pytest.mark.parametrize("compression", ["snappy", "none"])
@pytest.mark.parametrize("page_version", [1, 2])
def test_writer_round_trip(gp, tmp_path, compression, page_version):
    from sedona_gpuspatial import datagen, wkb
    inp = datagen.workload1(n_points=200000, n_polys=3000)
    rng = np.random.default_rng(page_version)
    for col, nulls in ((inp.probe, True), (inp.build, False)):
        validity = np.packbits(rng.random(len(col)) > 0.1, bitorder="little") if nulls else None
        c = wkb.WkbColumn(col.offsets, col.data, validity)
        path = str(tmp_path / "rt.parquet")
        gp.write_wkb(path, c, compression=compression, page_version=page_version,
                     row_group_rows=70000, page_bytes=1 << 18)
        with gp.GeoParquetFile(path) as f:
            got = gp.device_to_host(f.read_wkb())
        valid = (np.unpackbits(validity, bitorder="little")[:len(c)].astype(bool)
                 if nulls else np.ones(len(c), bool))
        off = col.offsets.astype(np.int64)
        keep = np.repeat(valid, np.diff(off))
        _assert_column(got, off, col.data[keep], valid)


def test_join_from_geoparquet(gp, tmp_path):
    """Build and probe sides read from GeoParquet give the pairs of the same
    columns passed directly."""
    from sedona_gpuspatial import capi, datagen
    inp = datagen.workload1(n_points=100000, n_polys=1000)
    pb, pp = str(tmp_path / "b.parquet"), str(tmp_path / "p.parquet")
    gp.write_wkb(pb, inp.build, compression="snappy")
    gp.write_wkb(pp, inp.probe, compression="snappy", page_version=2)
    j0 = capi.SpatialJoin()
    j0.build(inp.build)
    exp = gpu_util.pairs(*j0.probe(inp.probe, "intersects"))
    fb, fp = gp.GeoParquetFile(pb), gp.GeoParquetFile(pp)
    j = capi.SpatialJoin()
    import ctypes as C
    rc = capi.lib().SpjJoinBuildDevice(j.h, C.byref(fb.read_wkb()))
    assert rc == 0, capi.lib().SpjJoinLastError(j.h)
    db, dp, n = j.probe_device(fp.read_wkb(), "intersects")
    assert gpu_util.pairs(*gpu_util.device_pairs(db, dp, n)) == exp
    fb.close()
    fp.close()


def test_corrupt_page_is_an_error(gp, tmp_path):
    """A PLAIN length word that runs past its page fails the read with a
    message; the handle then reads a good file's column again."""
    from sedona_gpuspatial import datagen
    from sedona_gpuspatial.capi import GpuSpatialError
    inp = datagen.workload1(n_points=5000, n_polys=50)
    path = str(tmp_path / "c.parquet")
    gp.write_wkb(path, inp.build, compression="none")
    blob = bytearray(open(path, "rb").read())
    first = inp.build.value(0)
    at = bytes(blob).find(first)
    assert at > 4 and blob[at - 4:at] == np.uint32(len(first)).tobytes()
    blob[at - 4:at] = np.uint32(0x7FFFFFF0).tobytes()
    bad = str(tmp_path / "bad.parquet")
    open(bad, "wb").write(bytes(blob))
    with gp.GeoParquetFile(bad) as f:
        with pytest.raises(GpuSpatialError, match="PLAIN"):
            f.read_wkb()
    with gp.GeoParquetFile(path) as f:
        got = gp.device_to_host(f.read_wkb())
    assert np.array_equal(got.data, inp.build.data)


@pytest.mark.parametrize("page_version", [1, 2])
def test_device_matches_oracle(gp, oracle_lib, tmp_path, page_version):
    """The device reader against the CPU oracle's reading of the same file."""
    from sedona_gpuspatial import datagen, wkb
    inp = datagen.workload2(n_buildings=100000, n_zones=2000)
    col = inp.probe
    rng = np.random.default_rng(11)
    validity = np.packbits(rng.random(len(col)) > 0.05, bitorder="little")
    c = wkb.WkbColumn(col.offsets, col.data, validity)
    path = str(tmp_path / "o.parquet")
    gp.write_wkb(path, c, compression="snappy", page_version=page_version,
                 row_group_rows=40000, page_bytes=1 << 17)
    off, data, valid = oracle_lib.parquet_read(path)
    with gp.GeoParquetFile(path) as f:
        got = gp.device_to_host(f.read_wkb())
    _assert_column(got, off, data, valid)


@pytest.mark.parametrize("compression", ["snappy", "none"])
@pytest.mark.parametrize("kind", ["ragged", "decoys", "long", "mixed"])
def test_plain_values_of_unequal_lengths(gp, tmp_path, compression, kind):
    """The values' segments: starts that no guess finds (empty values, bytes
    that are no WKB), values that hold what looks like other values, values
    longer than a segment, pages of one value, nulls."""
    from sedona_gpuspatial import wkb
    rng = np.random.default_rng(len(kind))
    real = wkb.wkb_polygon([np.array([(0, 0), (3, 1), (2, 5), (0, 0)], np.float64)])

    def value(i):
        k = kind if kind != "mixed" else ["ragged", "decoys", "long", "real"][int(rng.integers(4))]
        if k == "ragged":
            return rng.integers(0, 256, int(rng.integers(0, 40)), dtype=np.uint8).tobytes()
        if k == "decoys":
            piece = len(real).to_bytes(4, "little") + real
            return rng.integers(0, 256, int(rng.integers(0, 9)), dtype=np.uint8).tobytes() + \
                piece * int(rng.integers(0, 60))
        if k == "long":
            return b"\x01" * int(rng.choice([0, 1, 4092, 4096, 4100, 30000]))
        return real
    n = 3000 if kind != "long" else 400
    vals = [value(i) for i in range(n)]
    off = np.zeros(n + 1, np.int64)
    off[1:] = np.cumsum([len(v) for v in vals])
    data = np.frombuffer(b"".join(vals), np.uint8)
    for nulls in (False, True):
        valid = rng.random(n) > 0.2 if nulls else np.ones(n, bool)
        c = wkb.WkbColumn(off, data, np.packbits(valid, bitorder="little") if nulls else None)
        path = str(tmp_path / "seg.parquet")
        gp.write_wkb(path, c, compression=compression, row_group_rows=n // 2 + 1,
                     page_bytes=1 << 15)
        with gp.GeoParquetFile(path) as f:
            got = gp.device_to_host(f.read_wkb())
        _assert_column(got, off, data[np.repeat(valid, np.diff(off))], valid)


@pytest.mark.parametrize("share", [0.02, 0.5, 0.98])
@pytest.mark.parametrize("compression", ["snappy", "none"])
def test_empty_values_before_a_guessed_one(gp, tmp_path, compression, share):
    """Segments that start with empty values, whose guess is the polygon behind
    them; runs of empty values over whole segments; a damaged length behind one."""
    from sedona_gpuspatial import capi, wkb
    rng = np.random.default_rng(int(share * 100))
    n = 20000
    lens = np.where(rng.random(n) < share, 0, 13 + 16 * rng.integers(4, 14, n))
    lens[5000:9000] = 0
    off = np.zeros(n + 1, np.int64)
    off[1:] = np.cumsum(lens)
    data = rng.integers(0, 256, int(off[-1]), dtype=np.uint8)
    at = off[:-1][lens > 0]
    data[at] = 1
    data[at[:, None] + np.arange(1, 5)] = (3, 0, 0, 0)
    path = str(tmp_path / "e.parquet")
    gp.write_wkb(path, wkb.WkbColumn(off, data, None), compression=compression, page_bytes=1 << 16)
    with gp.GeoParquetFile(path) as f:
        _assert_column(gp.device_to_host(f.read_wkb()), off, data, np.ones(n, bool))
    if compression == "none":
        raw = bytearray(open(path, "rb").read())
        k = raw.rfind(data[at[-1]:].tobytes()) - 4  # the last polygon's length word
        assert k > 0 and int.from_bytes(raw[k:k + 4], "little") == lens[lens > 0][-1]
        raw[k:k + 4] = (1 << 30).to_bytes(4, "little")
        open(path, "wb").write(raw)
        with gp.GeoParquetFile(path) as f, pytest.raises(capi.GpuSpatialError):
            f.read_wkb()


def test_files_share_page_locked_blocks(gp, tmp_path):
    """Threads that open, read and close files of several sizes one after the
    other: every read has its own bytes."""
    import threading
    from sedona_gpuspatial import wkb
    rng = np.random.default_rng(11)
    files = []
    for k, n in enumerate((3, 1000, 40000)):
        lens = rng.integers(0, 60, n)
        off = np.zeros(n + 1, np.int64)
        off[1:] = np.cumsum(lens)
        data = rng.integers(0, 256, int(off[-1]), dtype=np.uint8)
        path = str(tmp_path / f"{k}.parquet")
        gp.write_wkb(path, wkb.WkbColumn(off, data, None))
        files.append((path, off, data))
    bad = []

    def work(t):
        try:
            for i in range(12):
                path, off, data = files[(t + i) % len(files)]
                with gp.GeoParquetFile(path) as f:
                    got = gp.device_to_host(f.read_wkb())
                _assert_column(got, off, data, np.ones(len(off) - 1, bool))
        except BaseException as e:  # noqa: BLE001
            bad.append(e)
    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[0]


def test_trim_gives_back_page_locked_blocks(gp, tmp_path):
    """What closed files leave can be given back, what an open one uses cannot."""
    from sedona_gpuspatial import wkb
    path = str(tmp_path / "t.parquet")
    off = np.arange(0, 21 * 501, 21, dtype=np.int64)
    data = np.arange(off[-1]).astype(np.uint8)
    gp.write_wkb(path, wkb.WkbColumn(off, data, None))
    gp.trim()
    with gp.GeoParquetFile(path) as f:
        f.read_wkb()
        assert gp.trim() == 0
        _assert_column(gp.device_to_host(f.read_wkb()), off, data, np.ones(500, bool))
    assert os.path.getsize(path) // 2 < gp.trim() <= 256 << 20
    assert gp.trim() == 0
    with gp.GeoParquetFile(path) as f:
        _assert_column(gp.device_to_host(f.read_wkb()), off, data, np.ones(500, bool))
