"""Query groups with infinite coordinates, alone in their group (nothing finite lies in the lowest cells, where
such points are put) and among finite points: counts, harmonics, lists and neighbours are those of the
finite points alone. For harmonics the tolerance of the query-group tests, bonds of 0.4 and more:
(l + 1) 3e-6 / 0.4 absolute, 1e-5 relative."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

INF = np.float32(np.inf)


def system(freud, alone, flat=False, n=7000):
    rs = np.random.RandomState(3)
    L = 21.0 if not flat else 90.0
    box = freud.box.Box.square(L) if flat else freud.box.Box.cube(L)
    low = -0.2 if alone else -0.5
    pts = ((low + (0.5 - low) * rs.random_sample((n, 3))) * L).astype(np.float32)
    if flat:
        pts[:, 2] = 0
    k = 100
    for axis in range(2 if flat else 3):
        for value in (INF, -INF, np.float32(np.nan)):
            pts[k, axis] = value
            k += 1
    pts[k, :2] = INF
    pts[k + 1, :2] = [-INF, INF]
    return box, pts, np.isfinite(pts).all(axis=1)


@pytest.mark.parametrize("alone", [True, False])
@pytest.mark.parametrize("flat", [True, False])
@pytest.mark.parametrize("shell", [1, 2])
def test_histogram(freud, alone, flat, shell):
    box, pts, ok = system(freud, alone, flat)
    freud._lib.set_batch_config(shell, 8, 1)
    try:
        rdf = freud.density.RDF(40, 1.5)
        rdf.compute((box, pts))
        both = freud.density.RDF(40, 1.5)
        both.compute(freud.locality.FrameBatch([(box, pts), (box, pts[ok])]))
    finally:
        freud._lib.set_batch_config(0)
    want = O.rdf_counts_query(box, pts[ok], 40, 1.5)
    np.testing.assert_array_equal(rdf.bin_counts_u64, want)
    np.testing.assert_array_equal(both.bin_counts_u64, 2 * want)


@pytest.mark.parametrize("alone", [True, False])
@pytest.mark.parametrize("flat", [True, False])
@pytest.mark.parametrize("average", [False, True])
@pytest.mark.parametrize("n", [2500, 7000])  # (every pair; groups)
def test_harmonics(freud, alone, flat, average, n):
    box, pts, ok = system(freud, alone, flat, n)
    st = freud.order.Steinhardt(6, average=average)
    st.compute((box, pts), neighbors=dict(r_max=1.5, r_min=0.4))
    ij, d, _ = O.query(box, pts[ok], r_max=1.5, r_min=0.4, exclude_ii=True)
    o = O.steinhardt([6], box, pts[ok], ij, d, average=average)
    want = o["ql_ave" if average else "ql"][:, 0]
    np.testing.assert_allclose(np.asarray(st.ql, np.float64)[ok], want, rtol=1e-5, atol=7 * 3e-6 / 0.4 * (4 if flat else 1))


@pytest.mark.parametrize("alone", [True, False])
@pytest.mark.parametrize("flat", [True, False])
@pytest.mark.parametrize("k", [4, 20])
def test_neighbours(freud, alone, flat, k):
    box, pts, ok = system(freud, alone, flat)
    new = np.cumsum(ok) - 1
    nl = freud.locality.AABBQuery(box, pts).query(pts, dict(num_neighbors=k, exclude_ii=True)).toNeighborList()
    ij = np.asarray(nl[:])
    assert ok[ij[:, 1]].all() or not ok[ij[~ok[ij[:, 1]], 0]].any()
    keep = ok[ij[:, 0]]
    want, d, _ = O.query(box, pts[ok], num_neighbors=k, exclude_ii=True)
    np.testing.assert_array_equal(new[ij[keep]], want)
    np.testing.assert_array_equal(np.asarray(nl.distances)[keep], d)


@pytest.mark.parametrize("alone", [True, False])
@pytest.mark.parametrize("structure", ["aabb", "linkcell"])
def test_lists(freud, alone, structure):
    box, pts, ok = system(freud, alone, False, 30000)
    new = np.cumsum(ok) - 1
    nq = freud.locality.AABBQuery(box, pts) if structure == "aabb" else freud.locality.LinkCell(box, pts, 1.0)
    nl = nq.query(pts, dict(r_max=1.0, exclude_ii=True)).toNeighborList()
    want, d, _ = O.query(box, pts[ok], r_max=1.0, exclude_ii=True, arith=O.ARITH_AABB if structure == "aabb" else O.ARITH_WRAP)
    np.testing.assert_array_equal(new[np.asarray(nl[:])], want)
    np.testing.assert_array_equal(np.asarray(nl.distances), d)
