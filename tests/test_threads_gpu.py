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


# Every call that waits for its sizes, from eight threads with a stream each, new
# threads every round.
def test_threads_and_streams():
    g = _grid(sphere((61, 70, 83), 0.6))
    h = _grid(noise((20, 21, 33), 5, 0.1))
    sp = iso.SparseGrid([48, 48, 48])
    sp.populate(lambda p: p.norm(dim=-1) - 0.7)
    its = iso.get_intersection(h, 0.0, True)
    calls = [lambda: iso.marching_cubes(g), lambda: iso.dual_contouring(h), lambda: iso.marching_cubes(sp),
             lambda: iso.dual_contouring(sp), lambda: iso.dual_contouring(h, 0.0, its),
             lambda: (iso.get_intersection(g).get_points(),), lambda: iso.marching_cubes(h, method="lorensen"),
             lambda: iso.dual_contouring(g)]
    want = [[t.clone() for t in c()] for c in calls]
    torch.cuda.synchronize()
    bad = []

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for i in range(24):
                j = (k + i) % len(calls)
                got = calls[j]()
                if not all(torch.equal(a, b) for a, b in zip(got, want[j])):
                    bad.append((k, j))

    for _ in range(3):
        ts = [threading.Thread(target=work, args=(k,)) for k in range(8)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    assert not bad, bad
