"""Histograms of frames with points off the box and with coordinates that are not finite: no pair of
those is counted, and nothing is taken off for them. Against the oracle, bit for bit."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [400, 6000, 9000])  # every pair; the one-block grid; the general one
@pytest.mark.parametrize("shell", [0, 1, 2])
@pytest.mark.parametrize("exclude_ii", [True, False])
@pytest.mark.parametrize("off", [0, 1, 200])
def test_counts(freud, n, shell, exclude_ii, off):
    rs = np.random.RandomState(n + off)
    L = n ** (1 / 3.0)
    box = freud.box.Box.cube(L)
    pts = ((rs.random_sample((n, 3)) - 0.5) * L).astype(np.float32)
    pts[:off] += np.float32(L)
    pts[[390, 391, 392, 393, 394], [0, 1, 2, 0, 1]] = [np.nan, np.nan, np.nan, np.inf, -np.inf]
    pts[395] = np.nan
    freud._lib.set_batch_config(shell, 8, 1)
    try:
        rdf = freud.density.RDF(40, 1.5)
        rdf.compute((box, pts), neighbors=dict(r_max=1.5, exclude_ii=exclude_ii))
    finally:
        freud._lib.set_batch_config(0)
    finite = pts[np.isfinite(pts).all(axis=1)]
    np.testing.assert_array_equal(rdf.bin_counts_u64,
                                  O.rdf_counts_query(box, finite, 40, 1.5, exclude_ii=exclude_ii))
