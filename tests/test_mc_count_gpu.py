"""The sign bitmap, the count and the scan of marching cubes where their paths
change: words per row (rows that fill them or not), one or four words per
thread, rows on and off 16-byte boundaries, segments scanned by the last CTA or
by mc_scan, more than one round of listed words and one window of entries.
Checked against the oracle, bit for bit."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

import isoext_gb300 as iso  # noqa: E402
from helpers import assert_same_mesh, noise, sphere  # noqa: E402


def _check(oracle, vals, method):
    g = iso.UniformGrid(vals.shape)
    g.set_values(torch.from_numpy(np.ascontiguousarray(vals)).cuda())
    v, f = iso.marching_cubes(g, method=method)
    vo, fo, _ = oracle.mc_dense(vals, method=method)
    if v is None:
        assert len(fo) == 0
        return
    assert_same_mesh(v.cpu().numpy(), f.cpu().numpy(), vo, fo, str(vals.shape))


@pytest.mark.parametrize("nz", [2, 31, 32, 33, 64, 65, 96, 127, 129, 256, 257, 509, 512, 515, 1024, 1030, 1056])
def test_rows_of_every_kind(oracle, nz):
    # every second point inside: all words busy, every case, several rounds
    _check(oracle, noise((7, 5, nz), nz, 0.05), "nagae" if nz % 2 else "lorensen")


@pytest.mark.parametrize("shape", [(33, 31, 40), (64, 64, 2048), (65, 64, 2048), (83, 127, 802), (520, 510, 128)],
                         ids=str)
def test_segments_of_every_kind(oracle, shape):
    vals = sphere(shape, 0.8, center=(0.02, 0.01, -0.03)) if np.prod(shape) > 100000 else noise(shape, 1)
    _check(oracle, vals, "nagae")


@pytest.mark.parametrize("threads", [128, 256])
def test_count_threads(oracle, threads):
    from isoext_gb300 import tune

    old = tune.current()["mc.count_threads"]
    tune.set("mc.count_threads", threads)
    try:
        _check(oracle, noise((40, 41, 70), 2, 0.1), "lorensen")
        _check(oracle, sphere((150, 160, 480), 0.7), "nagae")
    finally:
        tune.set("mc.count_threads", old)
