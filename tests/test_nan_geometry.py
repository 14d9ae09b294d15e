"""Boys arguments that are not numbers (a shell position that is NaN): the class kernels take the far
row, so no row of the table is read at an index made from one (host build of the device code)."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "chronusq_public_b200", "csrc")
SOURCE = """
#include <cmath>
#define __device__
#define __host__
#define __forceinline__ inline
#define __align__(n) alignas(n)
struct double2 { double x, y; };
static inline int __double2int_rn(double x) { return (int)std::nearbyint(x); }
static inline double rsqrt(double x) { return 1.0 / std::sqrt(x); }
template <typename T> static inline T __ldg(const T *p) { return *p; }
#include "eri_common.cuh"
template <int L> void one(double s, double m, double R2, double *out) {
  const ClassArg a = class_arg<L>(s, m, R2);
  out[0] = a.far; out[1] = a.T; out[2] = boys_tfar(L); out[3] = a.y;
}
extern "C" void arg(int L, double s, double m, double R2, double *out) {
  switch (L) {
    case 0: return one<0>(s, m, R2, out);
    case 1: return one<1>(s, m, R2, out);
    case 2: return one<2>(s, m, R2, out);
    case 3: return one<3>(s, m, R2, out);
    case 4: return one<4>(s, m, R2, out);
    default: return one<5>(s, m, R2, out);
  }
}
"""


@pytest.fixture(scope="module")
def arg(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("class_arg")
    (d / "cuda_runtime.h").write_text("")
    (d / "a.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(d), "-I", CSRC, str(d / "a.cpp"), "-o",
                    str(d / "a.so")], check=True)
    f = ctypes.CDLL(str(d / "a.so")).arg
    f.argtypes = [ctypes.c_int] + [ctypes.c_double] * 3 + [ctypes.POINTER(ctypes.c_double)]
    f.restype = None

    def call(L, s, m, R2):
        out = (ctypes.c_double * 4)()
        f(L, s, m, R2, out)
        return tuple(out)
    return call


@pytest.mark.parametrize("L", range(6))
def test_far_row_for_what_is_not_a_number(arg, L):
    for s, m, R2 in ((2.0, 1.0, np.nan), (np.nan, np.nan, 1.0), (np.inf, np.inf, 0.0), (2.0, 1.0, np.inf)):
        far, T, tfar, y = arg(L, s, m, R2)
        assert far == 1.0 and T == tfar


@pytest.mark.parametrize("L", range(6))
def test_line_between_near_and_far(arg, L):
    tmax = {0: 36.0, 1: 40.0, 2: 44.0, 3: 47.0, 4: 50.0, 5: 52.0}[L]
    assert arg(L, 1.0, 1.0, tmax)[0] == 1.0
    far, T, tfar, y = arg(L, 1.0, 1.0, np.nextafter(tmax, 0.0))
    assert far == 0.0 and 0.0 <= T <= tmax and y == 1.0
    assert arg(L, 1.0, 1.0, 0.0)[:2] == (0.0, 0.0)
