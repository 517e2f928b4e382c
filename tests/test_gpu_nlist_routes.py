"""A ball query of the object's own points builds one grid, whichever order its list has."""

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
