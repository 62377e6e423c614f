"""The checked quotient of the device sweeps (dv_qdiv), restated on the CPU
with exact rational arithmetic: whatever the seed y0, a quotient that passes
the check is the correctly rounded a / b (the device repeats the others with
plain divisions), and with a seed as good as the hardware's nearly all pass.
"""
from fractions import Fraction as F

import numpy as np
import pytest

K = 1.0 + 2.0 ** -16


def rn(x: F) -> float:
    return x.numerator / x.denominator   # Python rounds this to nearest even


def fma(a, b, c):
    return rn(F(a) * F(b) + F(c))


def qdiv(a, b, y0):
    """(quotient, passed): the operations of dv_qdiv in its order."""
    e = fma(-b, y0, 1.0)
    qh = a * y0
    ql = fma(a, y0, -qh)
    qt = fma(qh, e, qh)
    s = fma(qh, e, ql)
    q = qh + fma(e * e, qt, s)
    r = fma(-b, q, a)
    t = fma(r, y0 * K, q)
    return q, t == q and abs(e) < 2.0 ** -17 and min(abs(a), abs(q)) >= 2.0 ** -960


def _pairs(kind, count, rng):
    m = lambda: float(rng.integers(1 << 52, 1 << 53))
    for _ in range(count):
        b = m()
        if kind == "random":
            a = m() * 2.0 ** int(rng.integers(-900, 900)) * (1 if rng.random() < 0.5 else -1)
        elif kind == "midpoint":   # a / b next to the middle of two doubles
            a = rn(F(b) * (F(int(m())) + F(1, 2))) * 2.0 ** -52
            a = float(np.nextafter(a, a * (0 if rng.random() < 0.5 else 2)))
        elif kind == "exact":      # a / b a double
            a = float(int(b) >> 30) * float(int(m()) >> 30)
            b = float(int(b) >> 30)
        else:                      # mantissas next to the top of a binade
            b = float((1 << 53) - int(rng.integers(1, 1 << 20)))
            a = float((1 << 53) - int(rng.integers(1, 1 << 53)))
        yield a, b


@pytest.mark.parametrize("kind", ["random", "midpoint", "exact", "top"])
@pytest.mark.parametrize("err", [2.0 ** -20, 2.0 ** -17.2, 2.0 ** -12, 1.0])
def test_accepted_quotient_is_correctly_rounded(kind, err):
    rng = np.random.default_rng(7)
    n = passed = 0
    for a, b in _pairs(kind, 400, rng):
        y0 = rn(F(1) / F(b)) * (1.0 + err * float(rng.uniform(-1, 1)))
        y0 = float(np.frombuffer(np.int64(np.float64(y0).view(np.int64) & ~0xffffffff).tobytes(),
                                 np.float64)[0])   # the seed's low word is zero
        q, ok = qdiv(a, b, y0)
        n += 1
        if ok:
            passed += 1
            assert q == a / b, (a, b, y0)
    if err <= 2.0 ** -20 and kind != "midpoint":
        assert passed >= 0.98 * n
    if err == 1.0:
        assert passed <= 0.05 * n
