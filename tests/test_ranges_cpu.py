"""The rows and segments that the weighted sums walk for a range of nodes
(csrc/tq_ranges.cuh, compiled for the host): every unit's reads lie inside the
range's values, no unit is empty and they cover the range once and in order, also where
the distances between a segment and the range leave 32 bits."""
import ctypes
import random
import subprocess

import pytest

from torchquad_gb300.build import CSRC

SHIM = """
#include "tq_ranges.cuh"
// 0, or 1 + the unit at which the walk leaves the range or skips a node
extern "C" int64_t check_walk(int64_t start, int64_t count, int64_t R, int64_t seg) {
  const tq::RowWalk w = tq::make_walk(start, count, R, seg);
  int64_t next = 0, u = 0;
  for (; u < w.units; ++u) {
    const tq::RowPart p = tq::row_part(w, u);
    if (p.lo < 0 || p.len < 0 || p.len > w.seg || p.j0 + p.len > R) return u + 1;
    if (p.lo >= p.len) return u + 1;  // a unit without nodes leaves a warp idle
    const int64_t first = p.r0 - w.start + p.j0 + p.lo;  // the value read first
    if (first != next || p.r0 != (w.row0 + p.row) * R) return u + 1;
    next += p.len - p.lo;
  }
  return next == count ? 0 : u + 1;
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("ranges")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC), "-o", str(d / "shim.so"),
                    str(d / "shim.cpp")], check=True)
    f = ctypes.CDLL(str(d / "shim.so")).check_walk
    f.restype = ctypes.c_int64
    f.argtypes = [ctypes.c_int64] * 4
    return f


G2 = 1 << 31


@pytest.mark.parametrize("start,count,R", [
    (0, 600_000_000, 3_000_000_000),                   # later segments lie more than 2^31 nodes ahead
    (2_400_000_000, 600_000_000, 3_000_000_000),       # earlier ones more than 2^31 nodes behind
    (G2 - 1, 3, 2 * G2 + 1), (G2 + 1, 2049, 2 * G2 + 1), (2 * G2 - 5, 6, 2 * G2 + 1), (0, 1, 2 * G2 + 1),
    (3 * G2 + 12345, 1_000_001, 4 * G2 + 1),
])
@pytest.mark.parametrize("seg", [2048, 512])
def test_rows_beyond_32_bits(check, start, count, R, seg):
    assert check(start, count, R, seg) == 0


def test_random_ranges(check):
    rng = random.Random(5)
    for _ in range(3000):
        seg = rng.choice([32, 64, 128, 256, 512, 1024, 2048])
        R = int(2 ** rng.uniform(1, 16)) + rng.randrange(3)
        total = R * rng.choice([1, 1, 2, 7, 40])
        start = rng.randrange(total)
        assert check(start, rng.randrange(1, total - start + 1), R, seg) == 0
