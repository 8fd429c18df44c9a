"""The room for the contraction's ranges (csrc/lv_kernels.cuh): whatever sizes the communities of a
level have -- degree bins configured so low that bin 7 starts at a few entries included -- the ranges
that `range_buckets` gives them all together fit `range_room`, each community's fit kRangeMax, and every
next-level id has one. Compiled with nvcc as host code (no GPU needed)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "louvain-fast-move-cuda_b200", "csrc")

SRC = r"""
#include <cstdio>
#include "lv_kernels.cuh"

using namespace lv;

static uint64_t rng = 88172645463325252ull;
static uint32_t below(uint32_t n) {
  rng ^= rng << 13; rng ^= rng >> 7; rng ^= rng << 17;
  return (uint32_t)((rng >> 11) % n);
}

// communities of [lo, hi] entries until the level's E are used up, among `ids` next-level vertices
static int level(uint32_t E, uint32_t lo, uint32_t hi, uint32_t ids) {
  uint64_t buckets = 0, left = E;
  while (left > 0) {
    uint64_t d = lo + (hi > lo ? below(hi - lo + 1) : 0);
    if (d > left) d = left;
    left -= d;
    const uint32_t nr = range_buckets((uint32_t)d, ids, kRangeLog);
    if (nr > 0) {
      const uint32_t log = range_log((uint32_t)d, ids);
      if (log > kRangeLog || nr > kRangeMax || ((uint64_t)nr << log) < ids) {
        std::printf("community of %u entries, %u ids: %u ranges of 2^%u\n", (uint32_t)d, ids, nr, log);
        return 1;
      }
    }
    buckets += nr;
  }
  if (buckets > range_room(E)) {
    std::printf("E=%u, communities of %u..%u entries, %u ids: %llu ranges, room for %u\n", E, lo, hi, ids,
                (unsigned long long)buckets, range_room(E));
    return 1;
  }
  return 0;
}

int main() {
  const uint32_t ids[] = {1, 2, 1000, 11500, 16384, 16385, 100000, 1u << 20, 1u << 24};
  const uint32_t size[][2] = {{1, 1}, {9, 9}, {65, 300}, {513, 1100}, {1000, 3100}, {2047, 2047}, {2048, 2048},
                              {2049, 2049}, {2040, 2060}, {4095, 4096}, {4097, 9000}, {100000, 400000}, {1u << 24, 1u << 26}};
  int bad = 0;
  for (uint32_t E : {1u << 24, (1u << 24) + 1u, 123456789u, 1u << 30})
    for (auto& z : size)
      if (E < 1u << 25 || z[0] > 1000)  // (few enough communities for a quick walk)
        for (uint32_t i : ids) bad += level(E, z[0], z[1], i);
  if (range_buckets(1u << 20, 100, 0) != 0) { std::printf("ranges where they are off\n"); ++bad; }
  if (!bad) std::printf("ok\n");
  return 0;
}
"""


def test_ranges_fit_their_room(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src = tmp_path / "ranges.cu"
    src.write_text(SRC)
    exe = tmp_path / "ranges"
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", CSRC, str(src), "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=300)
    assert out.stdout.strip() == "ok"
