"""Extractions while other host threads work: a launch parameter set meanwhile,
several threads and streams at once.  Results do not depend on either."""

import threading

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

import isoext_gb300 as iso  # noqa: E402
from helpers import noise, sphere  # noqa: E402
from isoext_gb300 import tune  # noqa: E402


def _grid(vals):
    g = iso.UniformGrid(vals.shape)
    g.set_values(torch.from_numpy(vals).cuda())
    return g


# one word per count thread with the segments scanned by the last CTA and by
# mc_scan; four words per thread
@pytest.mark.parametrize("vals", [noise((30, 31, 70), 3, 0.1), sphere((128, 130, 480), 0.7), sphere((200, 160, 500), 0.8)],
                         ids=["few", "many", "four"])
def test_count_threads_set_during_calls(vals):
    g = _grid(vals)
    old = tune.current()["mc.count_threads"]
    want = [t.clone() for t in iso.marching_cubes(g)]
    done = threading.Event()

    def flip():
        k = 0
        while not done.is_set():
            tune.set("mc.count_threads", (128, 256)[k & 1])
            k += 1

    t = threading.Thread(target=flip)
    t.start()
    try:
        for _ in range(200):
            v, f = iso.marching_cubes(g)
            assert torch.equal(v, want[0]) and torch.equal(f, want[1])
    finally:
        done.set()
        t.join()
        tune.set("mc.count_threads", old)
