"""The Sturm counts with checked quotients (dv_count_lat), the device function
itself compiled for the CPU, against plain loops with a / b, where a quotient
overflows, underflows or has a zero or subnormal divisor: in every row of a
chunk, its last one among them, whose successor belongs to the next chunk.
"""
import ctypes as C
import os
import re
import subprocess

import numpy as np
import pytest

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mr3smp_b200", "csrc",
                      "mr3_device.cuh")

HARNESS = r"""
#include <math.h>
#include <stdint.h>
#include <string.h>
#include <algorithm>
#include <type_traits>
using std::max; using std::min;
struct double2 { double x, y; };
#define __device__
#define __noinline__
#define __forceinline__ inline
#define __restrict__
static double __fma_rn(double a, double b, double c) { return fma(a, b, c); }
static double __dmul_rn(double a, double b) { return a * b; }
static double __dadd_rn(double a, double b) { return a + b; }
static int64_t bits(double x) { int64_t b; memcpy(&b, &x, 8); return b; }
// (a NaN's bits are the GPU's: one NaN)
static int __double2hiint(double x) { return x != x ? 0x7fffffff : (int)(bits(x) >> 32); }
static int __double2loint(double x) { return x != x ? -1 : (int)bits(x); }
static int d_imin(int a, int b) { return a < b ? a : b; }
static double dv_rcp_seed(double b) {   // rcp.approx.ftz: 20 bits, subnormals are zero
  if (fabs(b) < 2.2250738585072014e-308) b = copysign(0.0, b);
  double y = 1.0 / b;
  if (fabs(y) < 2.2250738585072014e-308) return copysign(0.0, y);
  if (isinf(y) || isnan(y)) return y;
  int64_t v = bits(y) & ~0xffffffffLL;
  memcpy(&y, &v, 8);
  return y;
}
@SOURCE@
template <int RULE> static int plain(int n, const double2 *tp, double pivmin, double c) {
  double t = tp[0].x - c;
  int cnt = 0;
  dv_count_row<RULE>(&t, &cnt, pivmin);
  for (int j = 1; j < n; j++) {
    t = dv_pivot<RULE>(tp[j].x, tp[j].y / t, c);
    dv_count_row<RULE>(&t, &cnt, pivmin);
  }
  return cnt;
}
extern "C" int count(int rule, int checked, int n, const double2 *tp, double pivmin, double c) {
  switch (rule) {
    case 0: return checked ? dv_count_lat<CNT_BISECT>(n, tp, pivmin, c) : plain<CNT_BISECT>(n, tp, pivmin, c);
    case 1: return checked ? dv_count_lat<CNT_IJOB1>(n, tp, pivmin, c) : plain<CNT_IJOB1>(n, tp, pivmin, c);
    case 2: return checked ? dv_count_lat<CNT_LARRC>(n, tp, 0.0, c) : plain<CNT_LARRC>(n, tp, 0.0, c);
    default: return checked ? dv_count_lat<CNT_LARRJ>(n, tp, 0.0, c) : plain<CNT_LARRJ>(n, tp, 0.0, c);
  }
}
extern "C" double quotient(double a, double b, int *failed) {   // one row as a chunk of its own
  qdiv_chk k;
  double qt;
  qdiv_begin(&k);
  const double q = dv_qdiv(a, b, dv_rcp_seed(b), &k, &qt);
  *failed = qdiv_failed(k, q);
  return q;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    src = open(HEADER).read()
    src = src[src.index("#define QDIV_KK"):src.index("// Guessed bisections.")]
    src = re.sub(r"static __device__ __forceinline__ double dv_rcp_seed\(.*?^}", "", src, flags=re.S | re.M)
    d = tmp_path_factory.mktemp("count")
    with open(d / "h.cpp", "w") as f:
        f.write(HARNESS.replace("@SOURCE@", src))
    so = str(d / "h.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-mfma", "-ffp-contract=off", "-fPIC", "-shared", "-o", so,
                    str(d / "h.cpp")], check=True)
    L = C.CDLL(so)
    L.count.argtypes = [C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_double, C.c_double]
    L.quotient.argtypes = [C.c_double, C.c_double, C.c_void_p]
    L.quotient.restype = C.c_double
    return L


@pytest.mark.parametrize("rule", ["bisect", "ijob1", "larrc", "larrj"])
def test_extreme_pivots(lib, rule):
    """A row whose pivot is tiny (its diagonal the point itself, the quotient
    before it next to underflow), then one whose quotient by it overflows."""
    r = ["bisect", "ijob1", "larrc", "larrj"].index(rule)
    rng = np.random.default_rng(3)
    tiny = float(np.finfo(float).tiny)
    for trial in range(2000):
        n, c = int(rng.integers(3, 40)), float(rng.choice([0.0, 0.25, -1.5]))
        tp = np.zeros((n, 2))
        tp[:, 0] = rng.uniform(-2, 2, n)
        tp[1:, 1] = rng.uniform(0, 2, n - 1) ** 2
        for _ in range(int(rng.integers(1, 4))):
            j = int(rng.integers(1, n))
            tp[j, 0] = c
            tp[j, 1] = float(rng.choice([0.0, tiny, 3 * tiny, 1e-320, 1e-300, 1e-285, 1e-280]))
            if j + 1 < n:
                tp[j + 1, 1] = float(rng.choice([1.0, 1e40, 1e100, 1e150]))
        piv = tiny * max(1.0, float(tp[:, 1].max()))
        got = lib.count(r, 1, n, tp.ctypes.data, piv, c)
        assert got == lib.count(r, 0, n, tp.ctypes.data, piv, c), (trial, n, tp)


def test_unchecked_quotients_are_those_of_the_division(lib):
    """Whatever is not recorded as failed is a / b, at the ends of the range too."""
    rng = np.random.default_rng(5)
    failed = C.c_int()
    passed = 0
    with np.errstate(all="ignore"):
        for _ in range(20000):
            a = np.float64(rng.uniform(1, 2) * 2.0 ** int(rng.integers(-1022, 1024)) * rng.choice([-1, 1]))
            b = np.float64(rng.uniform(1, 2) * 2.0 ** int(rng.integers(-1022, 1024)) * rng.choice([-1, 1]))
            q = lib.quotient(a, b, C.byref(failed))
            if not failed.value:
                passed += 1
                assert q == a / b, (a, b)
    assert passed > 8000
