"""The sort, the refinement list and the singletons' places made by one CTA,
at the sizes where the forms of many blocks take over: 2048 eigenvalues a
problem, 16384 rows and 4096 clusters a batch.  The results equal the
oracle's bit for bit on both sides of each."""
import pytest

import mr3smp_b200 as M
import oracle
from conftest import assert_same
from mr3smp_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _check(probs):
    for k, (p, r) in enumerate(zip(probs, M.mrrr_batched(probs))):
        assert_same(r, oracle.mrrr(p["jobz"], "A", p["D"], p["E"]), f"batch[{k}]")


@pytest.mark.parametrize("n", [2047, 2048, 2049])
def test_sort(n):
    small = wl.uniform(40, seed=3)
    D, E = wl.uniform(n, seed=n)
    _check([dict(jobz="V", range="A", D=small[0], E=small[1]),
            dict(jobz="N", range="A", D=D, E=E)])
    g, o = M.mrrr("V", "I", D, E, il=3, iu=60), oracle.mrrr("V", "I", D, E, il=3, iu=60)
    assert_same(g, o, f"n={n}")


@pytest.mark.parametrize("extra", [0, 1])
def test_refinement_list(extra):
    """128 problems of 128 rows with clusters, and one row more."""
    probs = []
    for k in range(128):
        n = 128 + (extra if k == 127 else 0)
        D, E = wl.wilkinson_plus(129)[:n].copy(), wl.uniform(n, seed=k)[1] * 0 + 1.0
        D[0] += k / 1024.0
        E[-1] = 0.0
        probs.append(dict(jobz="V", range="A", D=D, E=E))
    _check(probs)


@pytest.mark.parametrize("count", [4096, 4097])
def test_singleton_places(count):
    """A level 0 of `count` clusters (each problem's one block)."""
    probs = []
    for k in range(count):
        D, E = wl.uniform(2 + k % 5, seed=k)
        probs.append(dict(jobz="V", range="A", D=D, E=E))
    _check(probs)
