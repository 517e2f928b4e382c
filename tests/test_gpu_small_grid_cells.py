"""The one-block grid with cells of many points, where the block sorts all points: lists
against the oracle (a cell's points in index order are merged as sorted runs), sums that repeat to
the bit, and the time of the grid, which grew with the square of a cell's points."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def clusters(freud, n, cells):
    rs = np.random.RandomState(n + cells)
    box = freud.box.Box.cube(20.0)
    where = rs.randint(0, 20, (cells, 3))[rs.randint(0, cells, n)] - 9.5
    return box, (where + 0.4 * (rs.random_sample((n, 3)) - 0.5)).astype(np.float32)


# the sort has 64 words at least and any number of them; it is taken past 96 or 135 points in one cell, and of
# 8192 points in some 114 cells and fewer
@pytest.mark.parametrize("n, cells", [(1, 1), (63, 1), (64, 1), (65, 1), (66, 1), (127, 1), (129, 2), (450, 7), (640, 10),
                                      (1000, 1), (1024, 9), (1025, 13), (4097, 40), (8191, 90), (8192, 110), (8192, 120), (8192, 500), (96, 1), (97, 1), (135, 1), (136, 1), (3000, 3)])
@pytest.mark.parametrize("by_distance", [False, True])
def test_lists(freud, n, cells, by_distance):
    box, pts = clusters(freud, n, cells)
    for nq, arith in ((freud.locality.AABBQuery(box, pts), O.ARITH_AABB), (freud.locality.LinkCell(box, pts, 1.0), O.ARITH_WRAP)):
        args = dict(r_max=1.0, r_min=0.25, exclude_ii=True)
        nl = nq.query(pts, args).toNeighborList(sort_by_distance=by_distance)
        for a, b in zip((nl[:], nl.distances, nl.vectors), O.query(box, pts, arith=arith, sort_by_distance=by_distance, **args)):
            np.testing.assert_array_equal(np.asarray(a), b)


@pytest.mark.parametrize("n, cells", [(4000, 8), (6000, 60), (8192, 100)])
def test_order(freud, n, cells):
    box, pts = clusters(freud, n, cells)
    st = freud.order.Steinhardt(6, average=True, wl=True)
    first = None
    for _ in range(4):
        got = np.array(st.compute((box, pts), neighbors=dict(r_max=1.0, r_min=0.3)).ql)
        first = got if first is None else first
        np.testing.assert_array_equal(got, first)


def test_time(freud):
    """8192 points in one cell: the grid takes less than a quarter of a millisecond (0.4 to 1.2 by ranks)."""
    box, pts = clusters(freud, 8192, 1)
    best = np.inf
    for _ in range(5):
        nq = freud.locality.LinkCell(box, pts, 1.0)
        freud._lib.profile_enable(True)
        try:
            nq.query(pts, dict(r_max=1.0, r_min=0.9, exclude_ii=True)).toNeighborList(sort_by_distance=True)
            best = min(best, freud._lib.profile_report()["k_small_grid"][1])
        finally:
            freud._lib.profile_enable(False)
    assert best < 0.25
