"""Device memory kept for reuse: short-lived threads and callers' streams leave theirs to the next, all of
it goes back on request, and a call that failed leaves its buffers as usable as one that did not."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def used():
    import torch

    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def work(freud, seed=0, n=400000):
    """A list of some 26 million bonds (0.63 GB) and a histogram over it; its bonds and counts."""
    L = n ** (1 / 3.0)
    box = freud.box.Box.cube(L)
    pts = ((np.random.RandomState(seed).random_sample((n, 3)) - 0.5) * L).astype(np.float32)
    nq = freud.locality.AABBQuery(box, pts)
    nl = nq.query(pts, dict(r_max=2.5, exclude_ii=True)).toNeighborList()
    rdf = freud.density.RDF(50, 2.5)
    rdf.compute(nq, neighbors=nl)
    return len(nl), rdf.bin_counts_u64.tolist()


def test_threads(freud):
    got = []

    def one():
        t = threading.Thread(target=lambda: got.append(work(freud)))
        t.start()
        t.join()

    one()
    one()
    before = used()
    for _ in range(8):
        one()
    assert used() - before < 0.5e9
    assert got == 10 * got[:1]


def test_streams(freud):
    import torch

    def one():
        s = torch.cuda.Stream()
        freud._lib.set_stream(s.cuda_stream)
        try:
            work(freud)
        finally:
            freud._lib.set_stream(None)
        return s

    kept = [one(), one()]
    before = used()
    for _ in range(8):
        kept.append(one())
    assert used() - before < 0.5e9


def test_release(freud):
    work(freud)
    freud._lib.release_memory()
    before = used()
    n = work(freud)
    after = used()
    assert after - before > 0.4e9  # kept for the next list
    freud._lib.release_memory()
    assert abs(used() - before) < 0.1e9
    assert work(freud) == n


def test_after_an_error(freud):
    n = work(freud)
    box = freud.box.Box.cube(5.0)
    pts = np.zeros((10, 3), np.float32)
    for _ in range(3):
        with pytest.raises(RuntimeError):
            freud.locality.AABBQuery(box, pts).query(pts, dict(r_max=3.0)).toNeighborList()
        assert work(freud) == n
