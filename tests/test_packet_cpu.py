"""Host side of the packet refine's buffers: what a failed allocation leaves."""
import os
import subprocess

from sedona_gpuspatial import _build

SRC = r"""
#include <cstdio>
#include "packet.cuh"
int main() {
  spj::PacketBufs b;
  const uint64_t most = spj::PacketLimits(1ull << 40).chunks;
  for (uint64_t chunks : {most, (uint64_t)1}) {
    const bool ok = b.reserve(1000, chunks, chunks, 0);
    printf("%d %llu %llu\n", ok, (unsigned long long)b.chunk_cap, (unsigned long long)b.queue_cap);
  }
  const spj::PacketLimits small(1000);
  printf("%llu %llu\n", (unsigned long long)small.chunks, (unsigned long long)small.queue);
}
"""


def _run(tmp_path, source):
    """Compiles a program against the library and returns its output's lines."""
    lib = _build.build()
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(source)
    subprocess.run([_build.nvcc(), str(src), "-o", str(exe), lib, "-Xlinker",
                    "-rpath=" + os.path.dirname(lib)] + _build.NVCC_FLAGS, check=True)
    return subprocess.run([str(exe)], env=dict(os.environ, CUDA_VISIBLE_DEVICES=""), check=True,
                          capture_output=True, text=True).stdout.split("\n")


def test_failed_allocation_keeps_no_capacity(tmp_path):
    """Without a device every allocation fails: reserve says so, and neither
    the large nor the small request stays behind as a capacity."""
    out = _run(tmp_path, SRC)
    assert out[0] == out[1] == "0 0 0"
    assert out[2] == "3 62"  # chunks of 256 bytes, pairs of 16


RULE = r"""
#include <cstdio>
#include "engine.cuh"
using namespace spj;
int main() {
  struct Call { int predicate; bool points; uint64_t rows; PacketTree tree; };
  // (predicate, points, rows, {build rows, share, holes, crowd})
  const Call calls[] = {CALLS};
  for (const Call& c : calls) printf("%d\n", packet_pays(c.predicate, c.points, c.rows, c.tree));
}
"""
ZONES, STARS, TINY = 1.1e-3, 2.36e-5, 4.9e-7  # shares of the build rows' extent
# calls whose packets measured clearly slower (0) or faster (1) than their candidate pairs
CALLS = [
    ("kIntersects", 1, 65537, 50000, ZONES, 0, 0, 0), ("kIntersects", 1, 100000, 50000, ZONES, 0, 0, 0),
    ("kIntersects", 1, 200000, 50000, ZONES, 0, 0, 1), ("kContains", 1, 65537, 10000, ZONES, 0, 0, 0),
    ("kContains", 1, 140000, 10000, ZONES, 0, 0, 1), ("kIntersects", 1, 65537, 1000, ZONES, 0, 0, 1),
    ("kIntersects", 1, 65535, 1000, ZONES, 0, 0, 0), ("kIntersects", 1, 1000000, 10000, STARS, 0, 0, 1),
    ("kIntersects", 1, 65537, 50000, STARS, 0, 0, 0), ("kIntersects", 1, 1500000, 50000, TINY, 0, 0, 0),
    ("kIntersects", 1, 250000, 5000, TINY, 0, 0, 1), ("kDisjoint", 1, 80000, 50000, ZONES, 0, 0, 0),
    ("kIntersects", 0, 65537, 50000, ZONES, 0, 0, 1), ("kIntersects", 0, 2000000, 50000, ZONES, 0, 0, 1),
    ("kIntersects", 0, 1000000, 50000, STARS, 0, 0, 0), ("kIntersects", 0, 250000, 50000, TINY, 0, 0, 0),
    ("kIntersects", 0, 131072, 500, STARS, 0, 0, 1), ("kIntersects", 0, 131072, 10000, STARS, 0, 0, 1),
    ("kContains", 0, 8192, 50000, ZONES, 0, 0, 0), ("kContains", 0, 16000, 50000, ZONES, 0, 0, 0),
    ("kCovers", 0, 32000, 50000, ZONES, 0, 0, 1), ("kCovers", 0, 32000, 50000, STARS, 0, 0, 0),
    ("kContains", 0, 1000000, 50000, STARS, 0, 0, 1), ("kContains", 0, 300007, 20000, ZONES, 1, 0, 1),
    ("kContains", 0, 8192, 20000, ZONES, 1, 0, 0), ("kContains", 0, 16000, 20000, ZONES, 1, 0, 1),
    ("kTouches", 0, 8192, 50000, ZONES, 0, 0, 1), ("kTouches", 0, 8191, 50000, ZONES, 0, 0, 0),
    ("kTouches", 0, 8192, 5000, STARS, 0, 0, 1), ("kTouches", 0, 250000, 50000, TINY, 0, 0, 0),
    ("kWithin", 0, 8192, 50000, ZONES, 0, 0, 1), ("kEquals", 0, 32000, 1000, ZONES, 0, 0, 0),
    ("kCoveredBy", 0, 65000, 50000, TINY, 0, 0, 0),
    ("kPredDWithin", 1, 16000, 400000, 0, 0, 0.8, 0), ("kPredDWithin", 1, 16000, 400000, 0, 0, 3.0, 1),
    ("kPredDWithin", 1, 4000, 400000, 0, 0, 0.8, 1), ("kPredDWithin", 1, 20000, 5000, 0, 0, 0.1, 0),
    ("kPredDWithin", 1, 64000, 400000, 0, 0, 0.03, 1), ("kPredDWithin", 1, 2047, 5000, 0, 0, 50, 0),
    ("kPredDWithin", 1, 2048, 20000, 0, 0, 0.03, 1),
]


def test_packets_are_taken_where_they_measured_faster(tmp_path):
    rows = ", ".join("{%s, %s, %d, {%d, %r, %s, %r}}" % (
        p, "true" if pt else "false", n, nb, float(share), "true" if holes else "false", float(crowd))
        for p, pt, n, nb, share, holes, crowd, _ in CALLS)
    out = _run(tmp_path, RULE.replace("CALLS", rows))
    wrong = [c for c, o in zip(CALLS, out) if int(o) != c[-1]]
    assert not wrong
