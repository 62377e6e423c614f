"""dlarrf by a pair of lanes (dv_dlarrf<true>), the device function itself
compiled for the CPU: the two lanes are coroutines that run as far ahead of one
another as the warp operations let them, so that a lane which overwrites what
its partner has still to read is found.  Both lanes' shifts and the factors
are those of the one-lane form.
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
#include <ucontext.h>
#include <algorithm>
#include <type_traits>
#include <vector>
using std::max; using std::min; using std::isnan;
struct double2 { double x, y; };
#define __device__
#define __noinline__
#define __forceinline__ inline
#define __restrict__
#define MR3_EPS 2.220446049250313080847e-16
#define MR3_SAFMIN 2.225073858507201383090e-308
static double __fma_rn(double a, double b, double c) { return fma(a, b, c); }
static double __dmul_rn(double a, double b) { return a * b; }
static double __dadd_rn(double a, double b) { return a + b; }
static int64_t bits(double x) { int64_t b; memcpy(&b, &x, 8); return b; }
static int __double2hiint(double x) { return x != x ? 0x7fffffff : (int)(bits(x) >> 32); }
static int __double2loint(double x) { return x != x ? -1 : (int)bits(x); }
static int d_imin(int a, int b) { return a < b ? a : b; }
static int d_imax(int a, int b) { return a > b ? a : b; }
static double dv_rcp_seed(double b) {
  double y = 1.0 / b;
  if (isinf(y) || y != y) return y;
  int64_t v = bits(y) & ~0xffffffffLL;
  memcpy(&y, &v, 8);
  return y;
}
// ---- two lanes; `first` runs ahead
static ucontext_t g_main, g_ctx[2];
static double g_slot[2], g_old[2];
static int g_me, g_done[2], g_first, g_steps[2];
static bool g_pair;
struct { int x; } threadIdx;
static void meet(double v) {
  if (!g_pair) return;
  g_slot[g_me] = v;
  g_steps[g_me]++;
  swapcontext(&g_ctx[g_me], &g_main);
  threadIdx.x = g_me;
}
static double __shfl_sync(unsigned, double v, int src) { meet(v); return g_old[src & 1]; }
static int __shfl_sync(unsigned, int v, int src) { meet(v); return (int)g_old[src & 1]; }
static void __syncwarp(unsigned) { meet(0); }
static std::vector<double> g_growth[2];   // growth quantities that each lane has seen
static double seen(double x) { g_growth[g_pair ? g_me : 0].push_back(x); return x; }
@SOURCE@
struct In { int n, clend; const double2 *P, *Q; const double *w, *wgap, *werr; double spdiam, gl, gr, pivmin;
            double *dp, *lp, *wk; };
static In g_in;
static double g_sigma[2];
static int g_alt[2];
static void lane_main(int me) {
  g_me = me;
  threadIdx.x = me;
  const In &i = g_in;
  g_sigma[me] = dv_dlarrf<true>(i.n, i.P, i.Q, 1, i.clend, i.w, i.wgap, i.werr, i.spdiam, i.gl, i.gr,
                                i.pivmin, i.dp, i.lp, i.wk, 1, &g_alt[me]);
  g_done[me] = 1;
}
// 0: the lanes saw the same; 1: one left early; 2: growth quantities differ
extern "C" int pair(int first, int n, int clend, const double2 *P, const double2 *Q, const double *w,
                    const double *wgap, const double *werr, double spdiam, double gl, double gr,
                    double pivmin, double *dp, double *lp, double *wk, double *sigma, int *alt) {
  static std::vector<char> st[2] = {std::vector<char>(1 << 18), std::vector<char>(1 << 18)};
  g_in = {n, clend, P, Q, w, wgap, werr, spdiam, gl, gr, pivmin, dp, lp, wk};
  g_pair = true;
  for (int k = 0; k < 2; k++) {
    g_done[k] = g_steps[k] = 0;
    g_growth[k].clear();
    getcontext(&g_ctx[k]);
    g_ctx[k].uc_stack.ss_sp = st[k].data();
    g_ctx[k].uc_stack.ss_size = st[k].size();
    g_ctx[k].uc_link = &g_main;
    makecontext(&g_ctx[k], (void (*)())lane_main, 1, k);
  }
  while (!g_done[0] && !g_done[1]) {
    g_old[0] = g_slot[0]; g_old[1] = g_slot[1];
    for (int j = 0; j < 2; j++) {
      const int k = j ^ first;
      g_me = k;
      threadIdx.x = k;
      swapcontext(&g_main, &g_ctx[k]);
    }
  }
  for (int k = 0; k < 2; k++) { sigma[k] = g_sigma[k]; alt[k] = g_alt[k]; }
  return !(g_done[0] && g_done[1]) ? 1 : g_growth[0] != g_growth[1] ? 2 : 0;
}
extern "C" long one(int n, int clend, const double2 *P, const double2 *Q, const double *w,
                    const double *wgap, const double *werr, double spdiam, double gl, double gr,
                    double pivmin, double *dp, double *lp, double *wk, double *sigma, int *alt) {
  g_pair = false;
  g_growth[0].clear();
  threadIdx.x = 0;
  *sigma = dv_dlarrf<false>(n, P, Q, 1, clend, w, wgap, werr, spdiam, gl, gr, pivmin, dp, lp, wk, 1, alt);
  long c = 0;
  for (double x : g_growth[0]) c += x > 8.0;   // refused: another try follows
  return c;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    src = open(HEADER).read()
    a = src[src.index("#define QDIV_KK"):src.index("// Guessed bisections.")]
    a = re.sub(r"static __device__ __forceinline__ double dv_rcp_seed\(.*?^}", "", a, flags=re.S | re.M)
    b = src[src.index("static __device__ __forceinline__ double rrf_sweep("):
            src.index("// The factorisation T - sigma I = L D L^T of compute_root_rrr")]
    b = b.replace("  return tmp / (spdiam * sqrt(znm2));", "  return seen(tmp / (spdiam * sqrt(znm2)));")
    d = tmp_path_factory.mktemp("rrf")
    with open(d / "h.cpp", "w") as f:
        f.write(HARNESS.replace("@SOURCE@", a + b))
    so = str(d / "h.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-mfma", "-ffp-contract=off", "-fPIC", "-shared", "-o", so,
                    str(d / "h.cpp")], check=True)
    L = C.CDLL(so)
    L.one.restype = C.c_long
    return L


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("first", [0, 1])   # the lane that runs ahead
def test_pair_is_the_one_lane_form(lib, first):
    rng = np.random.default_rng(9)
    growth = alts = 0
    for trial in range(3000):
        n = int(rng.integers(4, 30))
        d, l = rng.uniform(0.1, 2.0, n), rng.uniform(-1.5, 1.5, n)
        l[-1] = 0.0
        if trial % 2:
            d *= rng.choice([-1.0, 1.0], n)
        P, Q = np.zeros((n, 2)), np.zeros((n, 2))
        P[:, 0], P[:, 1] = d, d * l * l
        Q[:, 0], Q[:, 1] = l, d * l
        M = np.eye(n) + np.diag(l[:-1], -1)
        w = np.linalg.eigvalsh(M @ np.diag(d) @ M.T)
        k = int(rng.integers(1, n - 1))
        wid = abs(w[k]) * 10.0 ** rng.uniform(-13, -5) + 1e-300
        ws, we = np.array([w[k], w[k] + wid]), np.array([wid, wid]) * 1e-3
        wg = np.array([wid, w[k + 1] - w[k]])
        # (a small diameter: the growth bounds are often exceeded)
        spd = float(w[-1] - w[0]) * 10.0 ** rng.uniform(-4, 0)
        args = (n, 2, _p(P), _p(Q), _p(ws), _p(wg), _p(we), C.c_double(spd),
                C.c_double(float(w[k] - w[k - 1])), C.c_double(float(w[k + 1] - w[k])), C.c_double(1e-300))
        o = [np.zeros(n), np.zeros(n), np.zeros(2 * n)]
        g = [np.zeros(n), np.zeros(n), np.zeros(2 * n)]
        so, sg, ao, ag = np.zeros(1), np.zeros(2), np.zeros(1, np.int32), np.zeros(2, np.int32)
        growth += lib.one(*args, *map(_p, o), _p(so), _p(ao)) > 0   # a try refused by its growth
        assert lib.pair(first, *args, *map(_p, g), _p(sg), _p(ag)) == 0, trial
        assert sg[0] == sg[1] == so[0] and ag[0] == ag[1] == ao[0], (trial, sg, so, ag, ao)
        f = 2 if ao[0] else 0
        if f:
            assert (g[2] == o[2]).all(), trial
        else:
            assert (g[0] == o[0]).all() and (g[1][:n - 1] == o[1][:n - 1]).all(), trial
        alts += int(ao[0])
    assert growth > 30 and alts > 30
