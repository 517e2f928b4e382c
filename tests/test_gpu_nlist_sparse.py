"""NeighborLists of a droplet in a box some thousand times r_max: the cells of r_max and those of
half of it are then the same grid (cells are limited to 2048 an axis and two a point), while the
droplet's groups have more candidates than a group holds and its queries go one at a time.
Against the block-per-cell kernels and the oracle, bit for bit."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

ARITH = {"linkcell": O.ARITH_WRAP, "aabb": O.ARITH_AABB}


def system(freud, L, droplet, sparse):
    rs = np.random.RandomState(droplet + int(L[0]))
    box = freud.box.Box(*L)
    pts = np.concatenate([(rs.random_sample((sparse, 3)) - 0.5) * np.array(L), 7.0 + 0.3 * rs.standard_normal((droplet, 3))])
    return box, rs.permutation(pts).astype(np.float32)


def lists(freud, structure, box, pts, queries=None, **args):
    q = pts if queries is None else queries
    args = dict(dict(exclude_ii=True), r_max=1.0, **args)
    want = O.query(box, pts, query_points=q, arith=ARITH[structure], **args)
    for which in (0, 1):
        freud._lib.set_count_kernel(which)
        try:
            nq = freud.locality.LinkCell(box, pts, 1.0) if structure == "linkcell" else freud.locality.AABBQuery(box, pts)
            for _ in range(2):  # (the second with its grids at hand)
                nl = nq.query(q, args).toNeighborList()
                for a, b in zip((nl[:], nl.distances, nl.vectors), want):
                    np.testing.assert_array_equal(np.asarray(a), b)
        finally:
            freud._lib.set_count_kernel(0)


@pytest.mark.parametrize("structure", ["linkcell", "aabb"])
@pytest.mark.parametrize("L, droplet, sparse", [((3000.0,) * 3, 1500, 3000), ((5000.0,) * 3, 2000, 3000),
                                                ((1130.0,) * 3, 1500, 3000), ((1148.0, 237.0, 231.0), 1500, 1132),
                                                ((1500.0,) * 3, 1100, 3400), ((3000.0,) * 3, 900, 3600)])
def test_droplet(freud, structure, L, droplet, sparse):
    box, pts = system(freud, L, droplet, sparse)
    lists(freud, structure, box, pts)
    lists(freud, structure, box, pts, queries=pts[::3] + np.float32(0.01), exclude_ii=False)
    lists(freud, structure, box, pts, r_min=0.4)


def test_not_finite(freud):
    box, pts = system(freud, (3000.0,) * 3, 40, 4460)
    pts[[5, 77, 800], [0, 1, 2]] = [np.nan, np.inf, -np.inf]
    lists(freud, "aabb", box, pts)
