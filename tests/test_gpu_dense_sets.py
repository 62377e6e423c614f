"""The buffer sets that the dense drivers keep between calls: calls of other
sizes and options after one another, and several threads at once, give the
results of a call alone bit for bit."""
import threading

import numpy as np
import pytest

import mr3smp_b200 as M

pytestmark = pytest.mark.gpu


def _matrix(n):
    A = np.random.default_rng(n).uniform(-1.0, 1.0, (n, n))
    return A + A.T


def _solve(n, uplo):
    r = M.dsyeig("V", "A", uplo, _matrix(n))
    assert r["info"] == 0 and r["m"] == n
    return r


@pytest.mark.parametrize("order", [(60, 130, 60, 7), (130, 1, 60, 130)])
def test_sizes_after_one_another_and_in_threads(order):
    alone = {}
    for n in (1, 7, 60, 130):
        alone[n] = _solve(n, "L")
    for n in order:
        g = _solve(n, "L")
        assert np.array_equal(g["W"], alone[n]["W"]) and np.array_equal(g["Z"], alone[n]["Z"])
    out = {}

    def work(k, n):
        out[k] = (n, _solve(n, "L"))
    ts = [threading.Thread(target=work, args=(k, n)) for k, n in enumerate(order + (60, 130))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert len(out) == len(ts)
    for n, g in out.values():
        assert np.array_equal(g["W"], alone[n]["W"]) and np.array_equal(g["Z"], alone[n]["Z"])
