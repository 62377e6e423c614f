"""A cluster cut by the index range whose computed values are equal.

When the blocks hold more eigenvalues than were asked for, the surplus is
taken from the largest values, the first of equal ones each time
(SRC/mrrr_val.c:515-626).  In a cluster of equal values that leaves a hole in
the local indices: here 188..204, 210..221 remain of 188..221 and il..iu ends
at 216.  The reference then refines the k-th value of the cluster as index
188 + k (dlarrb's offset, SRC/process_cluster.c:394-428), which is not its
own behind the hole; the device refines every value as its own index.  So the
eigenvectors of this cluster differ, both bases of nearly the same space;
everything else is equal bit for bit.
"""
import numpy as np
import pytest

import mr3smp_b200 as M
import oracle
from conftest import assert_same
from mr3smp_b200 import workloads as wl

pytestmark = pytest.mark.gpu

HOLED = slice(116, 145)   # the columns of the cluster with the hole


def test_only_the_cut_cluster_differs():
    D, E = wl.glued_wilkinson(17, 17, 1.0)
    E[16::17] = 1e-14
    E[-1] = 0.0
    g = M.mrrr("V", "I", D, E, il=72, iu=216)
    o = oracle.mrrr("V", "I", D, E, il=72, iu=216)
    assert g["m"] == 145
    Zg, Zo = g.pop("Z"), o.pop("Z")
    assert_same(g, o)
    same = np.ones(145, bool)
    same[HOLED] = False
    assert np.array_equal(Zg[:, same], Zo[:, same])
    assert wl.residual_orth(D, E, g["W"], Zg)[0] <= 10
    C = Zg[:, HOLED]
    # (orthonormal to 10 n eps, like any cluster's vectors)
    assert np.abs(C.T @ C - np.eye(C.shape[1])).max() <= 10 * len(D) * np.finfo(float).eps
