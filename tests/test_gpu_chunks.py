"""The sweeps in chunks of rows at the edges of their chunks: problem sizes
around multiples of 8 rows (the chunk of the checked quotients) and of 128
rows (the NaN blocks of dlaneg), clusters and zero shifts among them, with
every number of lanes per interval.  The results equal the oracle's bit for
bit."""
import numpy as np
import pytest

import mr3smp_b200 as M
import oracle
from conftest import assert_same
from mr3smp_b200 import workloads as wl

pytestmark = pytest.mark.gpu

SIZES = (2, 3, 7, 8, 9, 10, 15, 16, 17, 18, 25, 33, 127, 128, 129, 130, 136, 137, 265)


def _matrix(kind, n):
    if kind == "uniform":
        return wl.uniform(n, seed=900 + n)
    if kind == "wilkinson":   # pairs of close eigenvalues: child representations
        D, E = wl.wilkinson_plus(n | 1)[:n].copy(), np.ones(n)
        E[-1] = 0.0
        return D, E
    D, E = wl.one_two_one(n)   # zero pivots at the eigenvalue 2
    return D - 2.0, E


@pytest.mark.parametrize("lanes", ["1", "3", "5", "10", "32"])
@pytest.mark.parametrize("kind", ["uniform", "wilkinson", "121"])
def test_sizes_around_the_chunks(kind, lanes, monkeypatch):
    monkeypatch.setenv("MR3_TREE_LANES", lanes)
    for n in SIZES:
        D, E = _matrix(kind, n)
        for rng, kw in (("A", {}), ("I", dict(il=1 + n // 4, iu=max(1 + n // 4, n // 2)))):
            g, o = M.mrrr("V", rng, D, E, **kw), oracle.mrrr("V", rng, D, E, **kw)
            assert_same(g, o, f"{kind} n={n} {rng} lanes={lanes}")
        g, o = M.mrrr("N", "A", D, E), oracle.mrrr("N", "A", D, E)
        assert_same(g, o, f"{kind} n={n} N lanes={lanes}")


@pytest.mark.parametrize("finish_max", [None, "0", "700"])
def test_several_singletons_per_warp(finish_max, monkeypatch):
    """A list longer than the finish's warps (several groups of lanes per warp,
    bisections on the second list), finished from the level's start, in rounds
    only, and after some rounds."""
    if finish_max is not None:
        monkeypatch.setenv("MR3_FINISH_MAX", finish_max)
    probs = [dict(jobz="V", range="A", D=D, E=E)
             for D, E, _ in wl.mixed_batch(24, seed=77, nmin=5, nmax=500)]
    for n in (201, 335):
        D, E = wl.glued_wilkinson(5, n // 5 | 1, 1e-9)
        probs.append(dict(jobz="V", range="A", D=D, E=E))
    for k, (p, r) in enumerate(zip(probs, M.mrrr_batched(probs))):
        assert_same(r, oracle.mrrr("V", "A", p["D"], p["E"]), f"batch[{k}] {finish_max}")
