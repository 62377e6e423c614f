"""mr3_dense_release: the device memory that dense calls keep is given back, and
calls after it and beside it give the results of a call alone."""
import threading

import numpy as np
import pytest

import mr3smp_b200 as M

pytestmark = pytest.mark.gpu


def _solve(n):
    A = np.random.default_rng(n).uniform(-1.0, 1.0, (n, n))
    r = M.dsyeig("V", "A", "U", A + A.T)
    assert r["info"] == 0 and r["m"] == n
    return r


def test_release():
    import torch
    alone = _solve(900)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    assert M.dense_release() >= 1
    assert M.dense_release() == 0
    assert torch.cuda.mem_get_info()[0] - free0 >= 2 * 900 * 900 * 8   # A and Z at least
    again = _solve(900)
    assert np.array_equal(again["W"], alone["W"]) and np.array_equal(again["Z"], alone["Z"])


def test_release_beside_calls():
    alone = {n: _solve(n) for n in (80, 200)}
    out = []

    def work(n):
        for _ in range(5):
            r = _solve(n)
            out.append(np.array_equal(r["W"], alone[n]["W"]) and np.array_equal(r["Z"], alone[n]["Z"]))

    ts = [threading.Thread(target=work, args=(n,)) for n in (80, 200, 80)]
    for t in ts:
        t.start()
    while any(t.is_alive() for t in ts):
        M.dense_release()
        ts[0].join(0.005)
    for t in ts:
        t.join()
    assert len(out) == 15 and all(out)
