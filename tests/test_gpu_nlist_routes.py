"""A ball query of the object's own points builds one grid, whichever order its list has; and which
kernels list 2^22 points, whose groups sort keys of 64 bits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("structure", ["linkcell", "aabb"])
@pytest.mark.parametrize("by_distance", [False, True])
def test_one_grid(freud, structure, by_distance):
    n, L = 60000, 60000 ** (1 / 3.0)
    box = freud.box.Box.cube(L)
    pts = ((np.random.RandomState(1).random_sample((n, 3)) - 0.5) * L).astype(np.float32)
    nq = freud.locality.LinkCell(box, pts, 2.0) if structure == "linkcell" else freud.locality.AABBQuery(box, pts)
    freud._lib.profile_enable(True)
    try:
        nq.query(pts, dict(r_max=2.0, exclude_ii=True)).toNeighborList(sort_by_distance=by_distance)
        report = freud._lib.profile_report()
    finally:
        freud._lib.profile_enable(False)
    assert report["k_assign"][0] == 1


# groups of more than 512 candidates with 64-bit keys lose to the block-per-cell kernels
@pytest.mark.parametrize("n, r_max, groups", [((1 << 22) - 1, 2.9, True), (1 << 22, 2.9, False), (1 << 22, 1.5, True)])
@pytest.mark.parametrize("structure", ["linkcell", "aabb"])
def test_wide_keys(freud, structure, n, r_max, groups):
    L = n ** (1 / 3.0)
    box = freud.box.Box.cube(L)
    pts = ((np.random.RandomState(2).random_sample((n, 3)) - 0.5) * L).astype(np.float32)
    nq = freud.locality.LinkCell(box, pts, 2.0) if structure == "linkcell" else freud.locality.AABBQuery(box, pts)
    freud._lib.profile_enable(True)
    try:
        nl = nq.query(pts, dict(r_max=r_max, exclude_ii=True)).toNeighborList()
        report = freud._lib.profile_report()
    finally:
        freud._lib.profile_enable(False)
    assert ("k_nl_groups" in report) == groups
    mean = 4.0 / 3.0 * np.pi * r_max ** 3
    assert abs(len(nl) / n - mean) < 0.01 * mean
    assert np.asarray(nl.neighbor_counts).sum() == len(nl)
