"""Float-float harmonics of sets of l whose sums just fill the shared memory of a block: 46 to 48
sums a thread by two warps a block, 49 by the general kernel. Tolerance: each q_lm is the FP64 value
of its float32 bond vectors rounded once (2e-7 of the row's largest, with the oracle's own rounding)."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


# sums of the even orders: l / 2 + 1 each
@pytest.mark.parametrize("l, sums", [(0, 46), (2, 47), (4, 48), (6, 49)])
def test_sums(freud, l, sums):
    ls = [l, 26, 28, 30]
    assert sum(x // 2 + 1 for x in ls) == sums
    rs = np.random.RandomState(l)
    box = freud.box.Box.cube(6.0)
    pts = ((rs.random_sample((210, 3)) - 0.5) * 6).astype(np.float32)
    nl = freud.locality.AABBQuery(box, pts).query(pts, {"r_max": 1.4, "exclude_ii": True}).toNeighborList()
    st = freud.order.Steinhardt(ls, wl=True)
    st.compute((box, pts), neighbors=nl)
    o = O.steinhardt(ls, box, pts, np.array(nl[:]), np.array(nl.distances), wl=True)
    for k, h in enumerate(st.particle_harmonics):
        ok = np.isfinite(o["ql"][:, k])
        scale = np.abs(o["qlm"][k][ok]).max(axis=1, keepdims=True)
        assert np.all(np.abs(h[ok].astype(np.complex128) - o["qlm"][k][ok]) <= 2e-7 * scale + 2e-15)
