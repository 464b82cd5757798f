"""csrc/mhy_quot.h on the host: the branch-free reciprocal and quotient agree
with IEEE division bit for bit whenever they raise no flag, whatever the seed
inside its error bound, and raise the flag outside the documented range."""
import ctypes
import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
SRC = r'''
#include "mhy_quot.h"
#include <cstdint>
using namespace mhy;
static uint64_t s_;
static uint64_t rnd() { s_ += 0x9E3779B97F4A7C15ull; uint64_t z = s_; z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
                        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull; return z ^ (z >> 31); }
static double bits(uint64_t u) { double x; memcpy(&x, &u, 8); return x; }
static uint64_t ubits(double x) { uint64_t u; memcpy(&u, &x, 8); return u; }
// significand patterns: random, few bits, nearly all ones, short, just below a power of two
static double number(uint64_t u, int mode, int span) {
  uint64_t m = u & 0xfffffffffffffull;
  if (mode == 1) m &= 0xff;
  else if (mode == 2) m |= 0xfffffffffff00ull;
  else if (mode == 3) m &= 0xfffff00000000ull;
  else if (mode == 4) m = 0xfffffffffffffull - (m & 0xfff);
  const uint64_t e = 1023 + (int)((u >> 52) % (2 * span + 1)) - span;
  return bits((u & 0x8000000000000000ull) | e << 52 | m);
}
// mode bits choose the patterns and the exponent spans; returns wrong results among the unflagged ones
extern "C" long check(long n, uint64_t seed, int span, double seed_error, long* flagged) {
  s_ = seed; long wrong = 0; *flagged = 0;
  for (long i = 0; i < n; ++i) {
    const uint64_t m = rnd();
    const double y = number(rnd(), m % 5, span);
    double x = number(rnd(), (m >> 8) % 5, span);
    if ((m >> 20 & 31) == 0) x = (m >> 30 & 1) ? 0.0 : -0.0;
    const double d = ((double)(rnd() >> 11) * 0x1p-53 * 2 - 1) * seed_error;      // any seed within the bound
    unsigned bad = 0;
    const double r = rcp_from_seed(y, (1.0 / y) * (1.0 + d), bad);
    if (!bad && ubits(r) != ubits(1.0 / y)) ++wrong;
    const double q = quo_from_rcp(x, y, r, bad);
    if (!bad && ubits(q) != ubits(x / y)) ++wrong;
    if (bad) ++*flagged;
  }
  return wrong;
}
extern "C" unsigned flag(double x, double y) {
  unsigned bad = 0;
  const double r = rcp_from_seed(y, 1.0 / y, bad);
  quo_from_rcp(x, y, r, bad);
  return bad;
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("quot")
    (d / "q.cpp").write_text(SRC)
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-shared", "-fPIC",
                    f"-I{ROOT / 'arcane-benchs_b200' / 'csrc'}", str(d / "q.cpp"), "-o", str(d / "q.so")], check=True)
    lib = ctypes.CDLL(str(d / "q.so"))
    lib.check.argtypes = [ctypes.c_long, ctypes.c_uint64, ctypes.c_int, ctypes.c_double, ctypes.POINTER(ctypes.c_long)]
    lib.check.restype = ctypes.c_long
    lib.flag.argtypes = [ctypes.c_double, ctypes.c_double]
    lib.flag.restype = ctypes.c_uint
    return lib


@pytest.mark.parametrize("span", [0, 3, 40, 470])
@pytest.mark.parametrize("seed_error", [0.0, 2.0 ** -20, 0.999 * 2.0 ** -18])
def test_unflagged_results_are_ieee_division(lib, span, seed_error):
    flagged = ctypes.c_long()
    assert lib.check(2_000_000, 17 + span, span, seed_error, ctypes.byref(flagged)) == 0
    assert flagged.value < 0.03 * 2_000_000       # few quotients out of range


@pytest.mark.parametrize("x,y,expected", [
    (1.0, 3.0, 0), (0.0, 3.0, 0), (-0.0, 3.0, 0), (1.0, 0.0, 1), (0.0, 0.0, 1), (1.0, float("inf"), 1),
    (float("nan"), 1.0, 1), (1.0, float("nan"), 1), (float("inf"), 1.0, 1), (1e-300, 1.0, 1), (5e-324, 1.0, 1),
    (1.0, 1e-300, 1), (1e-200, 1e200, 1), (1e250, 1e-250, 1), (1.0, 1.0 - 2.0 ** -53, 0), (1e-280, 1e-280, 0)])
def test_flag(lib, x, y, expected):
    assert (lib.flag(x, y) != 0) == bool(expected)
