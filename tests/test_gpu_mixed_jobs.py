"""Batches that hold eigenvalues-only and count problems beside eigenvector
problems.  A problem without eigenvectors has neither Z nor Zsupp: when it
splits into blocks, its values lie block after block until they are sorted,
and the eigenvectors' order fix-up must pass it by.  The results equal the
oracle's bit for bit."""
import numpy as np
import pytest

import mr3smp_b200 as M
import oracle
from conftest import assert_same
from mr3smp_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _split(nb, bs, seed):
    """nb uncoupled blocks."""
    D, E = wl.uniform(nb * bs, seed=seed)
    E[bs - 1::bs] = 0.0
    return D, E


def _copies(nb, bs):
    """nb uncoupled copies of one block: its eigenvalues nb times, whose
    computed values may come out of order in the last bits."""
    D, E = wl.uniform(bs, seed=bs)
    return np.tile(D, nb), np.tile(E, nb)


def _problems(order):
    kinds = {
        "V": dict(jobz="V", range="A"), "N": dict(jobz="N", range="A"),
        "I": dict(jobz="N", range="I", il=5, iu=40), "C": dict(jobz="C", range="V", vl=-0.5, vu=0.7),
    }
    for k, c in enumerate(order):
        D, E = _copies(3 + k, 17) if k % 2 else _split(2 + k % 4, 31, seed=k)
        yield dict(kinds[c], D=D, E=E)


def _check(p, r, what):
    kw = {x: p[x] for x in ("vl", "vu", "il", "iu") if x in p}
    o = oracle.mrrr(p["jobz"], p["range"], p["D"], p["E"], **kw)
    if p["jobz"] == "C":
        assert r["info"] == o["info"] and r["m"] == o["m"], what
    else:
        assert_same(r, o, what)


@pytest.mark.parametrize("order", ["VN", "NV", "NVN", "VIV", "VNINVC", "CNVVNI", "NNNNNNNNV"])
def test_batch(order):
    probs = list(_problems(order))
    for k, (p, r) in enumerate(zip(probs, M.mrrr_batched(probs))):
        _check(p, r, f"{order}[{k}]")


def test_server():
    probs = list(_problems("VNNVNVVN" * 4))
    S = M.Server()
    try:
        tickets = [S.submit(p) for p in probs]
        res = [S.poll(t, wait=True)[0] for t in tickets]
    finally:
        S.close()
    for k, (p, r) in enumerate(zip(probs, res)):
        _check(p, r, f"request {k}")
