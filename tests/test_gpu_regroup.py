"""Intervals that end at very different steps within one warp: the groups left
move to more lanes.  Clusters next to the representation's shift, eigenvalues
alone and graded matrices, with every way to start (a thread per interval, 3,
4, 7, 10 and 32 lanes), small problems and large beside one another.  The
results equal the oracle's bit for bit."""
import numpy as np
import pytest

import mr3smp_b200 as M
import oracle
from conftest import assert_same
from mr3smp_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _matrix(kind, n):
    if kind == "glued":
        D, E = wl.glued_wilkinson(max(n // 21, 1), 21, 1e-8)
    elif kind == "graded":
        D, E = 10.0 ** (-8.0 * np.arange(n) / n), 10.0 ** (-8.0 * np.arange(n) / n) / 3
    else:
        D, E = wl.uniform(n, seed=40 + n)
    E = E.copy()
    E[-1] = 0.0
    return D, E


@pytest.mark.parametrize("lanes", ["1", "3", "4", "7", "10", "32"])
def test_batch(lanes, monkeypatch):
    monkeypatch.setenv("MR3_TREE_LANES", lanes)
    probs = []
    for n in (21, 33, 64, 65, 127, 210, 340, 501):
        for kind in ("glued", "graded", "uniform"):
            D, E = _matrix(kind, n)
            probs.append(dict(jobz="V" if n != 65 else "N", range="A", D=D, E=E, tryrac=n % 2))
    for k, (p, r) in enumerate(zip(probs, M.mrrr_batched(probs))):
        o = oracle.mrrr(p["jobz"], "A", p["D"], p["E"], tryrac=p["tryrac"])
        assert_same(r, o, f"lanes={lanes} batch[{k}]")


@pytest.mark.parametrize("count,nmin", [(40, 300), (330, 32), (500, 32)])
def test_singletons_bisections(count, nmin):
    """The singletons' bisections (several groups a warp, and in rounds): the
    state goes on in every lane of a group."""
    probs = [dict(jobz="V", range="A", D=D, E=E)
             for D, E, _ in wl.mixed_batch(count, seed=5, nmin=nmin, nmax=500)]
    for k, (p, r) in enumerate(zip(probs, M.mrrr_batched(probs))):
        assert_same(r, oracle.mrrr("V", "A", p["D"], p["E"]), f"batch[{k}]")
