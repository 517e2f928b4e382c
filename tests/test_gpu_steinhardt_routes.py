"""Which kernels a Steinhardt ball query runs, that it runs them once, and its values on every way,
in uniform systems and in droplets, whose cells of many points go in parts.

Tolerance as for the query groups: bond vectors carry about 3 roundings of magnitude L / 2 <= 16, on
bonds of 0.3 and more: (l + 1) 1e-5 absolute on q of order 1, plus 1e-5 relative."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def uniform(freud, n, seed=1):
    L = n ** (1 / 3.0)
    pts = ((np.random.RandomState(seed).random_sample((n, 3)) - 0.5) * L).astype(np.float32)
    return freud.box.Box.cube(L), pts


def droplet(freud, n, sigma, spread=0.0, L=30.0):
    rs = np.random.RandomState(n)
    m = int(n * spread)
    pts = np.concatenate([4.0 + sigma * rs.standard_normal((n - m, 3)), (rs.random_sample((m, 3)) - 0.5) * L])
    return freud.box.Box.cube(L), rs.permutation(pts).astype(np.float32)


def launches(freud, system, r_max, ls, average, st=None):
    """{kernel: launches} of a new object's compute."""
    st = st or freud.order.Steinhardt(ls, average=average)
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


ALL = [2, 4, 6, 8, 10, 12]
PAIRS, GROUPS, ARRAYS = "k_small_qlm", "k_frames_qlm", "k_qlm_ff2"


def ways(got):
    names = {name.split("<")[0] for name in got}
    return {way for way in (PAIRS, GROUPS, ARRAYS) if way in names}


# several l repeat the query, by pairs and by groups; bond arrays share it
@pytest.mark.parametrize("n, ls, r_max, average, way", [
    (1000, [6], 1.5, False, PAIRS), (1000, [6], 1.5, True, PAIRS), (500, [4, 6, 8, 10], 2.0, False, PAIRS),
    (2000, [4, 6, 8, 10], 1.5, True, ARRAYS), (2000, ALL, 2.5, True, ARRAYS), (5000, ALL, 1.5, False, ARRAYS),
    (20000, ALL, 2.0, True, ARRAYS), (8000, [4, 6, 8], 2.0, True, ARRAYS), (6000, [6], 1.5, False, GROUPS),
    (200000, [4, 6, 8], 1.5, False, GROUPS), (60000, [4, 6], 1.5, False, GROUPS)])
def test_ways(freud, n, ls, r_max, average, way):
    assert ways(launches(freud, uniform(freud, n), r_max, ls, average)) == {way}


# without averaging the fullest cell tells a droplet from a uniform system
@pytest.mark.parametrize("n, way", [(2000, PAIRS), (8000, GROUPS)])
def test_droplets_without_averaging(freud, n, way):
    got = launches(freud, droplet(freud, n, 1.0), 1.0, ALL, False)
    assert ways(got) == {way}


@pytest.mark.parametrize("system, r_max", [("uniform 700", 1.5), ("uniform 3000", 2.4), ("uniform 6000", 2.0),
                                           ("droplet 300", 1.0), ("droplet 2500", 0.8), ("droplet 6000", 0.6),
                                           ("half 5000", 0.9)])
@pytest.mark.parametrize("ls", [[6], [4, 6], [4, 6, 8], ALL])
@pytest.mark.parametrize("average, wl", [(False, False), (True, False), (True, True)])
def test_values(freud, system, r_max, ls, average, wl):
    kind, n = system.split()
    n = int(n)
    box, pts = (uniform(freud, n, seed=n) if kind == "uniform" else
                droplet(freud, n, 0.5 if n < 2000 else 0.8, 0.5 if kind == "half" else 0.0))
    ij, d, _ = O.query(box, pts, r_max=r_max, r_min=0.3, exclude_ii=True)
    o = O.steinhardt(ls, box, pts, ij, d, average=average)
    st = freud.order.Steinhardt(ls, average=average, wl=wl)
    st.compute((box, pts), neighbors={"r_max": r_max, "r_min": 0.3})
    tol = 1e-5 * (max(ls) + 1)
    want = o["ql_ave"] if average else o["ql"]
    np.testing.assert_allclose(np.asarray(st.ql, np.float64).reshape(want.shape), want, rtol=1e-5, atol=tol)
    if not wl:  # (the order is that of wl then)
        np.testing.assert_allclose(np.atleast_1d(st.order), o["order"], rtol=1e-5, atol=tol)
    h = st.particle_harmonics if len(ls) > 1 else [st.particle_harmonics]
    for k, l in enumerate(ls):
        power = np.sum(np.abs(h[k].astype(np.complex128)) ** 2, axis=1)
        np.testing.assert_allclose(np.sqrt(4 * np.pi / (2 * l + 1) * power), o["ql"][:, k], rtol=1e-5, atol=tol)


# cells of more than 128 points go in parts of 8
@pytest.mark.parametrize("n", [126, 128, 129, 136, 137, 500, 3000])
def test_cells_of_many_points(freud, n):
    box = freud.box.Box.cube(30.0)
    rs = np.random.RandomState(n)
    pts = np.concatenate([5.0 + 0.8 * rs.random_sample((n, 3)), (rs.random_sample((40, 3)) - 0.5) * 30]).astype(np.float32)
    pts = rs.permutation(pts)
    st = freud.order.Steinhardt([4, 6], average=True, wl=True)
    got = launches(freud, (box, pts), 1.0, None, None, st)
    assert "k_frames_ball<ONE>" in got
    ij, d, _ = O.query(box, pts, r_max=1.0, exclude_ii=True)
    o = O.steinhardt([4, 6], box, pts, ij, d, average=True)
    shortest = float(d.min())
    np.testing.assert_allclose(st.ql, o["ql_ave"], rtol=1e-5, atol=3e-6 * 7 / shortest)
