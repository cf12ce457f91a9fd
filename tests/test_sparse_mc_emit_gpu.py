"""Sparse marching cubes at the edges of its emit: chunks of 4096 cells full,
one short and one over; vertices and triangles past the 768 that one CTA stages;
cells with vertices on corners among cells without.  The oracle's mesh, exactly."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

import isoext_gb300 as iso  # noqa: E402
from helpers import assert_same_mesh, noise  # noqa: E402
from test_sparse_gpu import make_sparse, sparse_from_dense  # noqa: E402


@pytest.mark.parametrize("zeros", [0.0, 0.02, 0.4])
@pytest.mark.parametrize("n", [300, 4095, 4096, 4097, 8193])
def test_chunks_and_staging(oracle, n, zeros):
    vals = noise((3, 70, 70), n + int(100 * zeros), zeros)
    ids, cv = sparse_from_dense(vals, keep="all")
    ids, cv = ids[:n], cv[:n]
    for method in ("nagae", "lorensen"):
        v, f = iso.marching_cubes(make_sparse(vals.shape, ids, cv), method=method)
        vo, fo, _ = oracle.mc_sparse(ids, cv, vals.shape, method=method)
        assert_same_mesh(v.cpu().numpy(), f.cpu().numpy(), vo, fo, f"{n} {zeros} {method}")
