"""Range I of matrices with rows that are coupled to no other: such a row's
eigenvalue is its diagonal entry, which the search for the interval's end may
meet exactly.  Every range il..iu gives iu - il + 1 eigenpairs, and nothing is
written behind the iu - il + 1 columns of Z.  (The reference returns one more
where the end below il is such an eigenvalue.)
"""
import numpy as np
import pytest

import mr3smp_b200 as M
from mr3smp_b200 import workloads as wl

pytestmark = pytest.mark.gpu

MATRICES = {
    "diagonal": ([1.0, 0.0, -1.0], [0.0, 0.0, 0.0]),
    "integers": ([0.0, -2.0, 1.0, 0.0], [0.0, 1.0, -1.0, 0.0]),
    "two_blocks": ([3.0, -2.0, 3.0, 1.0, 3.0, 2.0, -1.0, 0.0, 0.0],
                   [1.0, -1.0, 0.0, -1.0, 0.0, -2.0, 1.0, 0.0, 0.0]),
    "equal_rows": ([2.0, 2.0, 2.0, 1.0, 2.0], [0.0, 0.0, 1.0, 0.0, 0.0]),
    "zeros": ([0.0] * 6, [0.0] * 6),
}


def _dense(D, E):
    return np.diag(D) + np.diag(E[:-1], 1) + np.diag(E[:-1], -1)


def _problems(name):
    D, E = (np.array(x) for x in MATRICES[name])
    n = len(D)
    for il in range(1, n + 1):
        for iu in range(il, n + 1):
            for jobz in "VN":
                yield dict(jobz=jobz, range="I", D=D, E=E, il=il, iu=iu)


def _check(p, info, m, W, Z=None):
    D, E, k = p["D"], p["E"], p["iu"] - p["il"] + 1
    w = np.linalg.eigvalsh(_dense(D, E))[p["il"] - 1:p["iu"]]
    assert info == 0 and m == k, (p, info, m)
    assert np.abs(W - w).max() <= 10 * len(D) * np.finfo(float).eps * max(1.0, np.abs(D).max()), p
    if Z is not None:
        res, orth = wl.residual_orth(D, E, W, Z) if np.abs(D).max() > 0 else (0.0, 0.0)
        assert res <= 10 and orth <= 10, p


@pytest.mark.parametrize("name", MATRICES)
def test_every_range(name):
    probs = list(_problems(name))
    for p, r in zip(probs, M.mrrr_batched(probs)):
        _check(p, r["info"], r["m"], r["W"], r.get("Z"))
    for p in probs[::3]:   # alone: the interval search by the whole CTA
        r = M.mrrr(p["jobz"], "I", p["D"], p["E"], il=p["il"], iu=p["iu"])
        _check(p, r["info"], r["m"], r["W"], r.get("Z"))


@pytest.mark.parametrize("name", MATRICES)
def test_nothing_behind_z(name):
    import torch
    probs, dev = [p for p in _problems(name) if p["jobz"] == "V"], []
    for p in probs:
        n, k = len(p["D"]), p["iu"] - p["il"] + 1
        dev.append(dict(p, D=torch.tensor(p["D"], device="cuda"), E=torch.tensor(p["E"], device="cuda"),
                        W=torch.zeros(n, dtype=torch.float64, device="cuda"),
                        Z=torch.full((n * k + 4 * n,), 7.0, dtype=torch.float64, device="cuda"),
                        Zsupp=torch.full((2 * k + 8,), 7, dtype=torch.int32, device="cuda")))
    rc, res = M.mrrr_batched_device(dev)
    torch.cuda.synchronize()
    assert rc == 0
    for p, d, r in zip(probs, dev, res):
        n, k = len(p["D"]), p["iu"] - p["il"] + 1
        Z = d["Z"].cpu().numpy()
        _check(p, r.info, r.m, d["W"].cpu().numpy()[:r.m], Z[:n * k].reshape(k, n).T)
        assert (Z[n * k:] == 7.0).all() and (d["Zsupp"][2 * k:] == 7).all(), p
