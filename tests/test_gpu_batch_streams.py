"""A batch used on a caller's stream has nothing to do with that stream afterwards: destroying it does
not wait for the stream's later work (nor touch a stream that may be gone)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["rdf", "steinhardt", "steinhardt wl"])
def test_destroy_does_not_wait(freud, what):
    import torch

    rs = np.random.RandomState(2)
    box = freud.box.Box.cube(20.0)
    frames = [(box, ((rs.random_sample((7000, 3)) - 0.5) * 20).astype(np.float32)) for _ in range(3)]
    # (its context and clock kernel exist before)
    torch.cuda._sleep(1000)
    user = torch.cuda.Stream()
    freud._lib.set_stream(user.cuda_stream)
    try:
        batch = freud.locality.FrameBatch(frames)
        if what == "rdf":  # bins of its own: the histogram's launch is tuned, on grids of either shell
            freud.density.RDF(83, 1.9).compute(batch, neighbors=dict(r_max=1.9))
        else:
            freud.order.Steinhardt(6, wl=what.endswith("wl")).compute(batch, neighbors=dict(r_max=1.4))
    finally:
        freud._lib.set_stream(None)
    with torch.cuda.stream(user):
        torch.cuda._sleep(600_000_000)  # about a third of a second
        after = torch.cuda.Event()
        after.record(user)
    del batch
    still_running = not after.query()
    torch.cuda.synchronize()
    assert still_running
