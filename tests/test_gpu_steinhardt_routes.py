"""Which kernels a Steinhardt ball query runs, and that it runs them once."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def uniform(freud, n, seed=1):
    L = n ** (1 / 3.0)
    pts = ((np.random.RandomState(seed).random_sample((n, 3)) - 0.5) * L).astype(np.float32)
    return freud.box.Box.cube(L), pts


def launches(freud, system, r_max, ls, average):
    """{kernel: launches} of a new object's compute."""
    st = freud.order.Steinhardt(ls, average=average)
    freud._lib.set_graphs(0)
    freud._lib.profile_enable(True)
    try:
        st.compute(system, neighbors={"r_max": r_max})
        report = freud._lib.profile_report()
    finally:
        freud._lib.profile_enable(False)
        freud._lib.set_graphs(1)
    return {name: count for name, (count, _) in report.items()}


# 20 to 200 bonds a point at density 1
@pytest.mark.parametrize("bonds", [20, 65, 130, 200])
def test_bond_lists_fit(freud, bonds):
    n = 200000
    got = launches(freud, uniform(freud, n), (bonds / 4.18879) ** (1 / 3.0), 6, True)
    assert got["k_frames_qlm<LIST>"] == 1


# averaging lists up to 64 neighbours a particle; the expected number decides, with four deviations
@pytest.mark.parametrize("n", [600, 2000, 3072])
@pytest.mark.parametrize("bonds, fits", [(14, True), (38, True), (41, False), (60, False), (113, False)])
def test_small_averaged(freud, n, bonds, fits):
    system = uniform(freud, n)
    got = launches(freud, system, (bonds / 4.18879) ** (1 / 3.0), 6, True)
    assert got.get("k_small_qlm", 0) == (1 if fits else 0)
    # without averaging nothing is listed
    assert launches(freud, system, (bonds / 4.18879) ** (1 / 3.0), 6, False).get("k_small_qlm", 0) == 1
