"""Sparse dual contouring in one call (iso_sparse_dc) against the sequence of calls
that a caller's intersection takes: the same mesh, bit for bit, on bands of
many tiles, missing neighbours, cells that disagree, vertices clipped onto their
cells' faces, ids past the lattice, NaN values and the retries."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

import isoext_gb300 as iso  # noqa: E402
from helpers import noise, sphere  # noqa: E402


def _grid(vals, ids, box=((-1,) * 3, (1,) * 3)):
    """Sparse grid of the given cells with corner values from a dense array."""
    nx, ny, nz = vals.shape
    g = iso.SparseGrid(vals.shape, *box)
    g.add_cells(torch.from_numpy(np.asarray(ids, np.int32)).cuda())
    i = g.get_cell_indices().long()
    x, y, z = i // ((ny - 1) * (nz - 1)), (i // (nz - 1)) % (ny - 1), i % (nz - 1)
    v = torch.from_numpy(vals).cuda()
    c = torch.arange(8, device="cuda")
    x, y, z = (a[:, None] + o for a, o in ((x, c >> 2), (y, (c >> 1) & 1), (z, c & 1)))
    g.set_values(v[x.clamp(max=nx - 1), y, z].contiguous())
    return g


def _both(g, level=0.0):
    v, f = iso.dual_contouring(g, level=level)
    its = iso.get_intersection(g, level=level, compute_normals=True)
    w, h = iso.dual_contouring(g, level=level, intersection=its)
    assert (v is None) == (w is None)
    if v is None:
        return 0
    assert v.shape == w.shape and f.shape == h.shape
    assert torch.equal(v.view(torch.int32), w.view(torch.int32)) and torch.equal(f, h)
    return len(f)


def _all(shape):
    return np.arange((shape[0] - 1) * (shape[1] - 1) * (shape[2] - 1))


def _cuboid(n):
    a = np.abs(np.linspace(-1, 1, n, dtype=np.float32))
    x, y, z = np.meshgrid(a - np.float32(0.5), a - np.float32(0.6), a - np.float32(0.55), indexing="ij")
    return np.maximum(x, np.maximum(y, z)).astype(np.float32)


@pytest.mark.parametrize("arith", ["nvcc", "host"])
@pytest.mark.parametrize("case", ["sphere", "noise", "dropped", "disagree", "cuboid", "thin", "past", "nan", "fine"])
def test_one_call_equals_the_sequence(case, arith):
    iso.set_arithmetic(arith)
    try:
        rng = np.random.default_rng(3)
        box = ((-1,) * 3, (1,) * 3)
        if case == "thin":
            vals = noise((2, 61, 33), 1)
        elif case == "cuboid":
            vals = _cuboid(48)
        elif case in ("noise", "nan", "disagree", "past"):
            vals = noise((21, 18, 37), 4, 0.1)
        elif case == "fine":  # coordinates that repeat: many vertices share positions
            vals = noise((9, 11, 40), 6)
            box = ((1.0, 1.0, 1.0), (1.0 + 2e-6, 1.0 + 3e-6, 1.0 + 2e-6))
        else:
            vals = sphere((70, 66, 58), 0.7, center=(0.02, -0.01, 0.03))
        if case == "nan":
            vals[rng.random(vals.shape) < 0.03] = np.nan
        ids = _all(vals.shape)
        if case == "dropped":
            ids = ids[rng.random(len(ids)) < 0.7]
        if case == "past":
            ids = np.concatenate([ids, ids[-1] + 1 + np.arange(300)])
        g = _grid(vals, ids, box)
        if case == "disagree":
            u = g.get_values()
            u[torch.rand(u.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(1)) < 0.05] *= -1.0
            g.set_values(u.contiguous())
        for level in (0.0, 0.03):
            faces = _both(g, level)
            assert faces or case in ("thin", "fine")
    finally:
        iso.set_arithmetic("nvcc")


def test_retries_reach_the_sizes():
    """Every cell active and more than one quad per cell: both capacities of the
    first attempt are too small."""
    vals = noise((40, 40, 40), 2)
    g = _grid(vals, _all(vals.shape))
    assert _both(g) > 2 * g.get_num_cells() // 4
    g._dc_sizes = {(g.get_num_cells(), 0.0): (10, 10)}
    assert _both(g)


def test_no_active_cell_gives_none():
    g = _grid(sphere((12, 12, 12), 0.5), np.arange(30))
    assert iso.dual_contouring(g, level=50.0) == (None, None)


@pytest.mark.parametrize("active", [511, 512, 513, 1023 * 512 + 1, 1024 * 512, 1024 * 512 + 1, 700_000])
def test_block_counts(active):
    """One block of active cells and up to the 1024 that the weld's last CTA scans
    by itself, and more (a launch of its own): noise, where every cell is active."""
    n = 100
    vals = noise((n, n, n), seed=active, zero_frac=0.02)
    corners = [vals[i:n - 1 + i, j:n - 1 + j, k:n - 1 + k] < 0 for i in (0, 1) for j in (0, 1) for k in (0, 1)]
    neg = sum(c.astype(np.int32) for c in corners).ravel()
    ids = np.flatnonzero((neg > 0) & (neg < 8))[:active]
    assert len(ids) == active
    assert _both(_grid(vals, ids)) > 0
