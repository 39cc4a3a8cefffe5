"""The sweep's quotient from a reciprocal, compiled for the host from the kernels' own source, against IEEE division: pairs whose
quotients lie next to a rounding boundary, and cells at the bounds within which the kernels use it."""

import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent.parent / "citrus_gb300" / "csrc" / "sweep.cu"

SHIM = r"""
#include <cmath>
#include <cstdint>
#include <cstring>
#define __device__
#define __forceinline__ inline
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fdiv_rn(float a, float b) { return a / b; }
static inline float __frcp_rn(float a) { return 1.0f / a; }
static inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
"""

DRIVER = r"""
static uint64_t state = 1;
static uint32_t rnd() { state = state * 6364136223846793005ull + 1442695040888963407ull; return (uint32_t)(state >> 32); }
static bool same(float a, float b) { return std::memcmp(&a, &b, 4) == 0; }

// mantissas a and b of 24 bits with t b = a 2^s + c for a t of 25 bits, odd: a / b is c / (b 2^s) away from the middle of two
// floats; s is 24 where a >= b and 25 where a < b. Times powers of two to the ends of the range of a.
extern "C" long near_midpoints(long pairs, long* tried) {
  long wrong = 0;
  *tried = 0;
  for (long n = 0; n < pairs; ++n) {
    uint32_t b = (1u << 23) | (rnd() & 0x7fffff) | 1;
    if (n % 4 == 0) b = (1u << 24) - 1 - 2 * (uint32_t)(n / 4 % 4096);
    if (n % 4 == 1) b = (1u << 23) + 1 + 2 * (uint32_t)(n / 4 % 4096);
    uint32_t inverse = b;
    for (int i = 0; i < 5; ++i) inverse *= 2 - b * inverse;  // of b modulo 2^32 (Newton)
    const int c = (int)(2 * (rnd() % 16)) - 15;              // odd, -15 to 15
    for (int s = 24; s <= 25; ++s) {
      const uint32_t low = ((uint32_t)c * inverse) & ((1u << s) - 1);
      const uint32_t t = s == 24 ? low | (1u << 24) : low;
      if (t < (1u << 24) || !(t & 1)) continue;
      const int64_t a = ((int64_t)t * b - c) >> s;
      if (a < (1 << 23) || a >= (1 << 24)) continue;
      const int exponents[4] = {-82, -23, 0, 35};              // a from 2e-18 to 6e17
      for (int e : exponents) {
        const float x = ldexpf((float)a, e), y = ldexpf((float)b, e + (int)(rnd() % 4));
        ++*tried;
        wrong += !same(quotient(x, y, 1.0f / y), x / y);
      }
    }
  }
  return wrong;
}

extern "C" long cells(long tries) {
  const float edge[8] = {0.f, kPlainMin, std::nextafter(kPlainMin, 1.f), kPlainMax, std::nextafter(kPlainMax, 0.f), 1.f,
                         std::nextafter(kPlainMin, 0.f), std::nextafter(kPlainMax, INFINITY)};
  long wrong = 0;
  for (long n = 0; n < tries; ++n) {
    float v[4];
    for (float& x : v)
      x = rnd() % 4 == 0 ? edge[rnd() % 8] : ldexpf((float)((1u << 23) | (rnd() & 0x7fffff)), -23 + (int)(rnd() % 120) - 60);
    if (v[0] + v[1] + v[2] == 0.f) continue;                 // no direction
    LaneCoef a, b;
    std::memset((void*)&a, 0, sizeof a);
    std::memset((void*)&b, 0, sizeof b);
    direction_coef(rnd() & 7, v[0], v[1], v[2], a);
    b = a;
    b.plain = false;                                         // divisions
    cell_coef(v[3], a);
    cell_coef(v[3], b);
    wrong += !(same(a.rdx, b.rdx) && same(a.rdy, b.rdy) && same(a.rdz, b.rdz) && same(a.rden, b.rden) &&
               same(a.qsx, b.qsx) && same(a.qsy, b.qsy) && same(a.qsz, b.qsz));
  }
  return wrong;
}
"""


@pytest.fixture(scope="module")
def lane(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not found")
    text = SOURCE.read_text()
    struct = text[text.index("struct LaneCoef"):]
    struct = struct[:struct.index("};") + 3]
    body = text[text.index("constexpr float kPlainMin"):text.index("// The lane of entry e, direction d and group g")]
    folder = tmp_path_factory.mktemp("quotient")
    (folder / "lane.cpp").write_text(SHIM + struct + body + DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(folder / "lane.so"),
                    str(folder / "lane.cpp")], check=True)
    return ctypes.CDLL(str(folder / "lane.so"))


def test_quotient_is_the_division_next_to_midpoints(lane):
    tried = ctypes.c_long()
    assert lane.near_midpoints(ctypes.c_long(2_000_000), ctypes.byref(tried)) == 0
    assert tried.value > 2_000_000


def test_cells_at_the_bounds_equal_divisions(lane):
    assert lane.cells(ctypes.c_long(2_000_000)) == 0
