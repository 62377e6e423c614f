"""Guessed bisections (dv_count_guess), restated on the CPU: the Sturm count
with its rounding errors does not decrease with the point, and a bisection
run with inaccurate counts and confirmed by exact counts at its two ends gives
the interval of the exact bisection bit for bit, however bad the guesses.
"""
import numpy as np
import pytest

from mr3smp_b200 import workloads as wl

PIV = float(np.finfo(np.float64).tiny)


def sturm(d, e2, c, pert=None):
    """dlaebz's count (odebz.f loop 90); pert: relative errors of the quotients."""
    t = d[0] - c
    cnt = 0
    if t <= PIV:
        cnt, t = 1, min(t, -PIV)
    for k in range(1, len(d)):
        q = e2[k - 1] / t
        if pert is not None:
            q *= 1.0 + pert[k]
        t = d[k] - q - c
        if t <= PIV:
            cnt += 1
            t = min(t, -PIV)
    return cnt


def bisect(count, j, a, b, reltol=1.5e-8, itmax=200):
    for _ in range(itmax):
        c = 0.5 * (a + b)
        if j <= count(c):
            b = c
        else:
            a = c
        if abs(b - a) < max(4 * PIV, reltol * max(abs(a), abs(b))):
            break
    return a, b


def _matrices():
    yield "uniform", wl.uniform(25, seed=3)
    yield "121", wl.one_two_one(17)
    yield "wilkinson", (wl.wilkinson_plus(21), np.r_[np.ones(20), 0.0])
    yield "glued", wl.glued_wilkinson(3, 9, 1e-9)


@pytest.mark.parametrize("name,T", list(_matrices()), ids=lambda x: x if isinstance(x, str) else "")
def test_counts_are_monotone(name, T):
    d, e = T
    e2 = e[:-1] ** 2
    w = np.linalg.eigvalsh(np.diag(d) + np.diag(e[:-1], 1) + np.diag(e[:-1], -1))
    for lam in w:   # points a few units in the last place around each eigenvalue
        x = [float(lam)]
        for _ in range(40):
            x.append(float(np.nextafter(x[-1], np.inf)))
        x = [lam - (y - lam) for y in x[:0:-1]] + x
        counts = [sturm(d, e2, c) for c in sorted(x)]
        assert all(p <= q for p, q in zip(counts, counts[1:])), (name, lam)


@pytest.mark.parametrize("err", [0.0, 1e-12, 1e-8, 1e-3, 1.0])
@pytest.mark.parametrize("name,T", list(_matrices()), ids=lambda x: x if isinstance(x, str) else "")
def test_confirmed_guess_is_the_exact_bisection(name, T, err):
    d, e = T
    e2 = e[:-1] ** 2
    rng = np.random.default_rng(5)
    r = np.abs(e) + np.r_[0.0, np.abs(e[:-1])]
    lo, hi = float((d - r).min()) - 1e-9, float((d + r).max()) + 1e-9
    confirmed = 0
    for j in range(1, len(d) + 1):
        pert = err * rng.uniform(-1, 1, len(d))
        a, b = bisect(lambda c: sturm(d, e2, c, pert), j, lo, hi)
        if sturm(d, e2, a) < j <= sturm(d, e2, b):
            confirmed += 1
            assert (a, b) == bisect(lambda c: sturm(d, e2, c), j, lo, hi), (name, j)
    if err <= 1e-12 and name == "uniform":
        assert confirmed >= len(d) - 1


def bracket_mid(l, r):
    if l < 0.0 < r:
        return 0.0
    if l >= 0.0:
        s = max(l, PIV)
        return float(np.sqrt(s) * np.sqrt(r)) if r > 4.0 * s else 0.5 * (l + r)
    return -bracket_mid(-r, -l)


@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_bracketed_walk_is_the_bisection(sign):
    """The walk of a long bisection from a bracket found at other points: the
    intervals of the bisection that counts at every midpoint."""
    g = 10.0 ** (-np.arange(24) * 11.0)
    d, e2 = sign * 3.0 * g, g[:-1] * g[1:]
    for j in range(1, 25):
        a0, b0 = -4.5, 4.5
        ref = bisect(lambda c: sturm(d, e2, c), j, a0, b0, itmax=1100)
        lo, hi = a0, b0
        counts = 0
        while hi - lo > 0.125 * max(4 * PIV, 1.5e-8 * max(abs(lo), abs(hi))):
            m = bracket_mid(lo, hi)
            if not lo < m < hi:
                break
            counts += 1
            if j <= sturm(d, e2, m):
                hi = m
            else:
                lo = m
        assert counts < 60

        def count(c):
            return j if c >= hi else j - 1 if c <= lo else sturm(d, e2, c)
        assert bisect(count, j, a0, b0, itmax=1100) == ref, j
