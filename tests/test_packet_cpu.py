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


def test_failed_allocation_keeps_no_capacity(tmp_path):
    """Without a device every allocation fails: reserve says so, and neither
    the large nor the small request stays behind as a capacity."""
    lib = _build.build()
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(SRC)
    subprocess.run([_build.nvcc(), str(src), "-o", str(exe), lib, "-Xlinker",
                    "-rpath=" + os.path.dirname(lib)] + _build.NVCC_FLAGS, check=True)
    out = subprocess.run([str(exe)], env=dict(os.environ, CUDA_VISIBLE_DEVICES=""), check=True,
                         capture_output=True, text=True).stdout.split("\n")
    assert out[0] == out[1] == "0 0 0"
    assert out[2] == "3 62"  # chunks of 256 bytes, pairs of 16
