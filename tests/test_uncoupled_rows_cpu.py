"""Range I where the search for eigenvalue il - 1 ends at the value of an
uncoupled row: the reference's order takes that row's eigenvalue although its
count has it below il, one more than iu - il + 1 in all.  The rule of the device
(k_blocks) takes a row's value exactly where the counts at the two ends say it
lies between them.
"""
import numpy as np
import pytest

import oracle

PIV = float(np.finfo(float).tiny)


def counted(d, c):
    """Whether the count at c has a 1x1 block's value below c (odebz.f loop 90)."""
    return d - c <= PIV


def taken(d, wl, wu):
    return not (d - wl <= PIV) and d - wu <= PIV


def taken_by_reference(d, wl, wu):   # SRC/mrrr_val.c:340-412
    return d + PIV > wl and d - PIV <= wu


def test_the_reference_takes_one_too_many():
    r = oracle.mrrr("V", "I", np.array([1.0, 0.0, -1.0]), np.zeros(3), il=3, iu=3)
    assert r["info"] == 0 and r["m"] == 2 and list(r["W"]) == [0.0, 1.0]
    assert counted(0.0, 0.0) and taken_by_reference(0.0, 0.0, 1.0)


@pytest.mark.parametrize("wl,wu", [(0.0, 1.0), (-1.0, 0.0), (1.0, 1.5), (-PIV, PIV), (0.0, 3 * PIV)])
def test_taken_where_the_counts_differ(wl, wu):
    points = [-1.0, -PIV, -5e-324, 0.0, -0.0, 5e-324, PIV, 2 * PIV, 4 * PIV, 1.0, 1.5]
    for x in (wl, wu):
        points += [x - PIV, x + PIV, float(np.nextafter(x, -9)), float(np.nextafter(x, 9))]
    for d in points:
        assert taken(d, wl, wu) == (counted(d, wu) and not counted(d, wl)), d
