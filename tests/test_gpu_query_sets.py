"""Few query points of their own against many points: ball lists, nearest neighbours and RDF
against the oracle, bit for bit. The query points are put into the cells of the points' grid, of
which there are up to two a point and so many times more than the query points: the
one-block build of small grids takes at most 2 x 8192 + 64 cells, the general build the others."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def system(n, m, flat=False):
    rs = np.random.RandomState(n % 1000 + m)
    L = n ** (1 / 2.0 if flat else 1 / 3.0)
    pts = ((rs.random_sample((n, 3)) - 0.5) * L).astype(np.float32)
    queries = ((rs.random_sample((m, 3)) - 0.5) * L).astype(np.float32)
    if flat:
        pts[:, 2] = queries[:, 2] = 0
    return L, pts, queries


def same(nl, want):
    for a, b in zip((nl[:], nl.distances, nl.vectors), want):
        np.testing.assert_array_equal(np.asarray(a), b)


# 8192 query points are the limit of the one-block build by points; 16448 cells that by cells:
# at r_max 1 and cells of r_max 8242 points have 20^3 cells, 16500 25^3 = 15625, 18000 26^3 = 17576
@pytest.mark.parametrize("n", [8242, 16500, 18000, 60000, 250000])
@pytest.mark.parametrize("m", [1, 100, 8192, 8193])
@pytest.mark.parametrize("flat", [False, True])
def test_few_queries(freud, n, m, flat):
    L, pts, queries = system(n, m, flat)
    box = freud.box.Box.square(L) if flat else freud.box.Box.cube(L)
    for nq, arith in ((freud.locality.AABBQuery(box, pts), O.ARITH_AABB),
                      (freud.locality.LinkCell(box, pts, 1.0), O.ARITH_WRAP)):
        same(nq.query(queries, dict(r_max=1.0)).toNeighborList(),
             O.query(box, pts, query_points=queries, r_max=1.0, arith=arith))
        same(nq.query(queries, dict(r_max=1.0)).toNeighborList(sort_by_distance=True),
             O.query(box, pts, query_points=queries, r_max=1.0, arith=arith, sort_by_distance=True))
        rdf = freud.density.RDF(40, 1.0)
        rdf.compute(nq, query_points=queries, neighbors=dict(r_max=1.0, exclude_ii=False))
        np.testing.assert_array_equal(
            rdf.bin_counts_u64,
            O.rdf_counts_query(box, pts, 40, 1.0, query_points=queries, exclude_ii=False, arith=arith))


@pytest.mark.parametrize("n", [8242, 60000, 250000])
@pytest.mark.parametrize("m", [1, 100, 8192])
@pytest.mark.parametrize("k", [4, 40])
def test_few_queries_nearest(freud, n, m, k):
    L, pts, queries = system(n, m)
    box = freud.box.Box.cube(L)
    same(freud.locality.AABBQuery(box, pts).query(queries, dict(num_neighbors=k)).toNeighborList(),
         O.query(box, pts, query_points=queries, num_neighbors=k))
