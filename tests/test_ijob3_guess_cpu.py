"""The guessed interval searches of dlaebz IJOB=3 (dv_ijob3_tree), the device
function itself compiled for the CPU: its source is taken out of the header,
lanes run as coroutines that meet at every warp or CTA operation, and the
guessed counts are exact counts at a point a little off, so that midpoints
next to an eigenvalue are guessed wrongly.  Whatever the guesses, the interval
and its counts are the sequential loop's, bit for bit; so they are when a
point closes the interval.
"""
import ctypes as C
import os
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "mr3smp_b200", "csrc", "mr3_device.cuh")

HARNESS = r"""
#include <math.h>
#include <ucontext.h>
#include <algorithm>
#include <vector>
struct double2 { double x, y; };
static double fmin_(double a, double b) { return a < b ? a : b; }
static int count_at(int n, const double2 *tp, double pivmin, double c) {   // odebz.f loop 90
  double t = tp[0].x - c;
  int cnt = 0;
  if (t <= pivmin) { cnt = 1; t = fmin_(t, -pivmin); }
  for (int j = 1; j < n; j++) {
    t = tp[j].x - tp[j].y / t - c;
    if (t <= pivmin) { cnt++; t = fmin_(t, -pivmin); }
  }
  return cnt;
}
static double g_off;         // the guesses: counts at points this far away
static long g_guess, g_exact;
enum { CNT_BISECT };
static int dv_count_guess(int n, const double2 *tp, double pivmin, double c) {
  g_guess++;
  return count_at(n, tp, pivmin, c + g_off);
}
template <int R> static int dv_count_lat(int n, const double2 *tp, double pivmin, double c) {
  g_exact++;
  return count_at(n, tp, pivmin, c);
}
// ---- lanes as coroutines
static int g_T;                          // threads of the CTA (or 32: a warp)
static ucontext_t g_main;
static std::vector<ucontext_t> g_ctx;
static std::vector<int> g_done;
static int g_me;
static std::vector<long long> g_slot, g_old;
struct { int x; } threadIdx;
static void meet(long long v) {          // every lane gets here, then all go on
  g_slot[g_me] = v;
  swapcontext(&g_ctx[g_me], &g_main);
  threadIdx.x = g_me;
}
static int __shfl_sync(unsigned, int v, int src) {
  const int w = g_me & ~31;
  meet(v);
  return (int)g_old[w + (src & 31)];
}
static int __any_sync(unsigned, int p) {
  const int w = g_me & ~31;
  meet(p != 0);
  for (int k = 0; k < 32 && w + k < g_T; k++) if (g_old[w + k]) return 1;
  return 0;
}
static int __syncthreads_or(int p) {
  meet(p != 0);
  for (int k = 0; k < g_T; k++) if (g_old[k]) return 1;
  return 0;
}
static void __syncthreads() { meet(0); }
static int __clz(int x) { return x ? __builtin_clz((unsigned)x) : 32; }
#define __device__
#define __noinline__
#define __forceinline__ inline
#define __restrict__
@SOURCE@
struct Walk { int n; const double2 *tp; double pivmin, abstol, reltol; int nitmax, nval; double c, a, b;
              int na, nb, L; int *cnt; double ra, rb; int rna, rnb; };
static Walk *g_walks;                    // one per group
static void lane_main(int me) {
  g_me = me;
  threadIdx.x = me;
  Walk &w = g_walks[me / g_walks[0].L];
  double a = w.a, b = w.b;
  int na = w.na, nb = w.nb;
  dv_ijob3_tree(w.L, w.cnt, w.n, w.tp, w.pivmin, w.abstol, w.reltol, w.nitmax, w.nval, w.c,
                count_at(w.n, w.tp, w.pivmin, w.c), &a, &b, &na, &nb);
  if (me % w.L == 0) { w.ra = a; w.rb = b; w.rna = na; w.rnb = nb; }
  g_done[me] = 1;
}
// T threads in groups of L, group g searching for nval[g] from the point c[g]
extern "C" void run(int T, int L, int cta, int n, const double2 *tp, double pivmin, double abstol,
                    double reltol, int nitmax, const int *nval, const double *c, double a, double b,
                    double off, double *rab, int *rnn, long *counts) {
  static std::vector<std::vector<char>> stacks;
  std::vector<int> cnt(T);
  std::vector<Walk> walks(T / L);
  for (int g = 0; g < T / L; g++)
    walks[g] = {n, tp, pivmin, abstol, reltol, nitmax, nval[g], c[g], a, b, -1, n + 1, L,
                cta ? cnt.data() : nullptr, 0, 0, 0, 0};
  g_T = T; g_off = off; g_walks = walks.data(); g_guess = g_exact = 0;
  g_ctx.resize(T); g_done.assign(T, 0); g_slot.assign(T, 0);
  while ((int)stacks.size() < T) stacks.emplace_back(1 << 16);
  for (int k = 0; k < T; k++) {
    getcontext(&g_ctx[k]);
    g_ctx[k].uc_stack.ss_sp = stacks[k].data();
    g_ctx[k].uc_stack.ss_size = stacks[k].size();
    g_ctx[k].uc_link = &g_main;
    makecontext(&g_ctx[k], (void (*)())lane_main, 1, k);
  }
  for (bool more = true; more;) {
    more = false;
    g_old = g_slot;
    for (int k = 0; k < T; k++)
      if (!g_done[k]) {
        g_me = k;
        threadIdx.x = k;
        swapcontext(&g_main, &g_ctx[k]);
        more |= !g_done[k];
      }
  }
  for (int g = 0; g < T / L; g++) {
    rab[2 * g] = walks[g].ra; rab[2 * g + 1] = walks[g].rb;
    rnn[2 * g] = walks[g].rna; rnn[2 * g + 1] = walks[g].rnb;
  }
  counts[0] = g_guess; counts[1] = g_exact;
}
// the sequential loop (odebz.f IJOB=3)
extern "C" void loop(int n, const double2 *tp, double pivmin, double abstol, double reltol, int nitmax,
                     int nval, double c, double a, double b, double *rab, int *rnn) {
  int na = -1, nb = n + 1;
  for (int it = 1; it <= nitmax; it++) {
    const int k = count_at(n, tp, pivmin, c);
    if (k <= nval) { a = c; na = k; }
    if (k >= nval) { b = c; nb = k; }
    if (fabs(b - a) < fmax(fmax(abstol, pivmin), reltol * fmax(fabs(a), fabs(b))) || na >= nb) break;
    c = 0.5 * (a + b);
  }
  rab[0] = a; rab[1] = b; rnn[0] = na; rnn[1] = nb;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    src = open(HEADER).read()
    parts = [re.search(r"^static __device__ __forceinline__ bool ijob3_step\(.*?^}", src, re.S | re.M),
             re.search(r"^#define IJOB3_WIDTH.*?$", src, re.M),
             re.search(r"^static __device__ __noinline__ void dv_ijob3_tree\(.*?^}", src, re.S | re.M)]
    d = tmp_path_factory.mktemp("ijob3")
    cpp, so = str(d / "h.cpp"), str(d / "h.so")
    with open(cpp, "w") as f:
        f.write(HARNESS.replace("@SOURCE@", "\n".join(p.group(0) for p in parts)))
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-o", so, cpp],
                   check=True)
    return C.CDLL(so)


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def _problems():
    rng = np.random.default_rng(11)
    for k in range(60):
        n = int(rng.integers(4, 14))
        if k % 3 == 0:
            d, e = np.full(n, 2.0), np.ones(n - 1)
        elif k % 3 == 1:
            d, e = np.abs(np.arange(n) - n // 2).astype(float), np.ones(n - 1)
        else:
            d, e = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n - 1)
        w = np.linalg.eigvalsh(np.diag(d) + np.diag(e, 1) + np.diag(e, -1))
        # ends whose first midpoints lie next to an eigenvalue
        lam = float(w[int(rng.integers(n))])
        r = float(max(w[-1] - lam, lam - w[0]) + rng.uniform(0.5, 1.5))
        shift = float(rng.choice([0.0, 1e-14, -1e-14, 3e-12]))
        yield n, d, e, lam - r + shift, lam + r, float(rng.choice([1, -1]) * 10.0 ** rng.uniform(-15, -9))


@pytest.mark.parametrize("T,L,cta", [(32, 16, 0), (32, 32, 0), (128, 64, 1), (256, 128, 1)])
def test_guessed_search_is_the_sequential_loop(lib, T, L, cta):
    piv, eps = float(np.finfo(float).tiny), float(np.finfo(float).eps)
    G = T // L
    closed = 0
    for n, d, e, a, b, off in _problems():
        tp = np.zeros((n, 2))
        tp[:, 0] = d
        tp[1:, 1] = e * e
        for nval in range(0, n + 1, 1 if T == 32 else 3):
            nv = np.array([(nval + g) % (n + 1) for g in range(G)], np.int32)
            c = np.array([a if v < n // 2 else b for v in nv])
            for nitmax in (5, 90):
                rab, rnn, counts = np.zeros(2 * G), np.zeros(2 * G, np.int32), np.zeros(2, np.int64)
                lib.run(T, L, cta, n, _p(tp), C.c_double(piv), C.c_double(4 * piv), C.c_double(4 * eps),
                        nitmax, _p(nv), _p(c), C.c_double(a), C.c_double(b), C.c_double(off), _p(rab),
                        _p(rnn), _p(counts))
                for g in range(G):
                    sab, snn = np.zeros(2), np.zeros(2, np.int32)
                    lib.loop(n, _p(tp), C.c_double(piv), C.c_double(4 * piv), C.c_double(4 * eps),
                             nitmax, int(nv[g]), C.c_double(c[g]), C.c_double(a), C.c_double(b),
                             _p(sab), _p(snn))
                    assert (rab[2 * g:2 * g + 2] == sab).all() and (rnn[2 * g:2 * g + 2] == snn).all(), \
                        (n, nval, g, nitmax, off, rab, sab, rnn, snn)
                    closed += snn[0] == snn[1]
    assert closed > 50   # searches that a point closed are among them
