"""csrc/mhy_quot.h on the host: a quotient formed with a plain reciprocal
(rcp_checked, the sweeps of several environments) raises the flag for every
denominator outside the documented range, also where the numerator is zero,
and agrees with IEEE division where it raises none."""
import ctypes
import math
import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
SRC = r'''
#include "mhy_quot.h"
extern "C" double quotient(double x, double y, unsigned* flag) {
  *flag = 0;
  const double r = mhy::rcp_checked(y, *flag);
  return mhy::quo_from_rcp(x, y, r, *flag);
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
    lib.quotient.argtypes = [ctypes.c_double, ctypes.c_double, ctypes.POINTER(ctypes.c_uint)]
    lib.quotient.restype = ctypes.c_double
    return lib


@pytest.mark.parametrize("x", [0.0, -0.0, 1.0, 5e-324, 2.0 ** 1000, math.inf, math.nan])
@pytest.mark.parametrize("y", [0.0, 5e-324, 2.0 ** -1025, 2.0 ** -960, 2.0 ** 960, 2.0 ** 1022, 2.0 ** 1023, math.inf, math.nan])
def test_a_denominator_out_of_range_raises_the_flag(lib, x, y):
    flag = ctypes.c_uint()
    for s in (1.0, -1.0):
        lib.quotient(x, s * y, ctypes.byref(flag))
        assert flag.value != 0, (x, s * y)


@pytest.mark.parametrize("x", [0.0, -0.0, 1.0, -3.0, 2.0 ** -400])
@pytest.mark.parametrize("y", [2.0 ** -550, 3.0, 1.0 - 2.0 ** -53, -7.0, 2.0 ** 500])
def test_what_raises_none_is_ieee_division(lib, x, y):
    flag = ctypes.c_uint()
    q = lib.quotient(x, y, ctypes.byref(flag))
    assert flag.value == 0
    assert q == x / y and math.copysign(1.0, q) == math.copysign(1.0, x / y)
