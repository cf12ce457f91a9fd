"""The cell numbering of dense dual contouring (dc_cells) and the one-call paths
with and without a caller's intersection, against the sequence of calls (cells
by word, hash weld): the same bits, at the edges of words, segments and scans."""

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

import isoext_gb300 as iso  # noqa: E402
from helpers import noise, sphere  # noqa: E402
from isoext_gb300 import _ffi, dc  # noqa: E402


def _grid(vals, lo=(-1, -1, -1), hi=(1, 1, 1)):
    g = iso.UniformGrid(vals.shape, lo, hi)
    g.set_values(torch.from_numpy(np.ascontiguousarray(vals)).cuda())
    return g


def _reference_intersection(g, level):
    """points, normals, cells, offsets of iso_dc_classify + iso_dc_intersect."""
    lib = _ffi.lib()
    nx, ny, nz = g.shape
    st = torch.cuda.current_stream().cuda_stream
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    ws = torch.empty(int(lib.iso_dc_workspace_size(nx, ny, nz)), dtype=torch.uint8, device="cuda")
    counts = torch.zeros(2, dtype=torch.int64, device="cuda")
    _ffi.check(lib.iso_dc_classify(p(g._values), nx, ny, nz, level, p(ws), ws.numel(), p(counts), st))
    A, K = counts.tolist()
    points, normals = (torch.empty((K, 3), dtype=torch.float32, device="cuda") for _ in range(2))
    cells, offs = (torch.empty(n, dtype=torch.int32, device="cuda") for n in (A, A + 1))
    _ffi.check(lib.iso_dc_intersect(p(g._values), nx, ny, nz, _ffi.fvec3(g.aabb_min), _ffi.fvec3(g.aabb_max), level,
                                    p(ws), A, K, p(points), p(normals), p(cells), p(offs), st))
    return points, normals, cells, offs


def _same(a, b):
    return a.shape == b.shape and torch.equal(a.view(torch.int32), b.view(torch.int32))


SHAPES = [(2, 2, 2), (2, 3, 31), (3, 2, 32), (5, 9, 33), (17, 16, 64), (9, 31, 129), (40, 50, 127),
          (64, 64, 2048),   # 2^18 point words: one word per thread
          (65, 64, 2048),   # four, rows on 16-byte boundaries
          (83, 127, 802),   # four, rows off them
          (520, 510, 128)]  # more segments than one CTA scans


@pytest.mark.parametrize("arith", ["nvcc", "host"])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_one_call_paths_equal_the_sequence(shape, arith):
    iso.set_arithmetic(arith)
    try:
        big = np.prod(shape) > 100000
        vals = sphere(shape, 0.8, center=(0.02, 0.01, -0.03)) if big else noise(shape, int(np.prod(shape)), 0.1)
        g = _grid(vals)
        for level in (0.0, 0.125):
            ref = _reference_intersection(g, level)
            for normals in (False, True):
                its = iso.get_intersection(g, level=level, compute_normals=normals)
                got = [its.get_points(), its._normals, its._cells, its._offsets]
                assert all(_same(x, y) for x, y in zip(got, ref) if x is not None)
                v, f = iso.dual_contouring(g, level=level, intersection=its)
                w, h = dc._dc_sequence(g, its, 1e-2, 1e-6) if its._cells.numel() else (None, None)
                u, e = iso.dual_contouring(g, level=level)
                assert (v is None) == (w is None) == (u is None)
                if v is not None:
                    assert _same(v, w) and torch.equal(f, h) and _same(v, u) and torch.equal(f, e)
    finally:
        iso.set_arithmetic("nvcc")


def _cuboid(shape, half=0.5, lo=(-1, -1, -1), hi=(1, 1, 1)):
    ax = [np.abs(np.linspace(-1, 1, n)) - half for n in shape]
    q = np.stack(np.meshgrid(*ax, indexing="ij"), -1)
    return (np.linalg.norm(np.maximum(q, 0), axis=-1) + np.minimum(q.max(-1), 0)).astype(np.float32)


@pytest.mark.parametrize("case", ["cuboid", "zeros", "repeated_coords"])
def test_local_weld_equals_the_hash_weld(case):
    """Vertices clipped to their cells' faces, crossings on grid points, and
    coordinates that repeat: the inputs on which the weld has vertices to merge."""
    lo, hi = (-1, -1, -1), (1, 1, 1)
    if case == "zeros":
        vals = noise((26, 22, 30), seed=9, zero_frac=0.3)
    elif case == "cuboid":
        vals = _cuboid((33, 29, 31))
    else:
        lo, hi = (1000.0, -1.0, 1000.0), (1000.001, 1.0, 1000.002)
        vals = _cuboid((24, 20, 28), 0.6)
    g = _grid(vals, lo, hi)
    its = iso.get_intersection(g, compute_normals=True)
    v, f = iso.dual_contouring(g, intersection=its)
    u, e = iso.dual_contouring(g)
    w, h = dc._dc_sequence(g, its, 1e-2, 1e-6)
    assert _same(v, w) and torch.equal(f, h) and _same(u, w) and torch.equal(e, h)


def test_caller_normals_equal_the_sequence():
    """Normals that push vertices out of their cells."""
    g = _grid(sphere((40, 33, 45), 0.7))
    its = iso.get_intersection(g)
    n = torch.zeros_like(its.get_points())
    n[:, 0] = 1.0
    n[::3, 1] = 3.0
    n[1::5, 2] = -2.0
    its.set_normals(n)
    v, f = iso.dual_contouring(g, intersection=its)
    w, h = dc._dc_sequence(g, its, 1e-2, 1e-6)
    assert _same(v, w) and torch.equal(f, h)


def test_values_changed_since_the_intersection():
    """As many active cells elsewhere, or another number of them: the call falls
    back to the sequence (whose quads follow the grid's values now)."""
    vals = sphere((30, 30, 30), 0.5, center=(0.2, 0.0, 0.0))
    g = _grid(vals)
    its = iso.get_intersection(g, compute_normals=True)
    v, f = iso.dual_contouring(g, intersection=its)
    g.set_values(torch.from_numpy(np.ascontiguousarray(vals[::-1])).cuda())
    assert dc._dc_given(g, its, 1e-2, 1e-6) is None
    w, h = iso.dual_contouring(g, intersection=its)
    assert h.shape == f.shape
    g.set_values(torch.from_numpy(sphere((30, 30, 30), 0.3)).cuda())
    assert dc._dc_given(g, its, 1e-2, 1e-6) is None


def test_intersection_retries_reach_the_sizes():
    vals = noise((24, 25, 26), 3)
    g = _grid(vals)
    key = ((24, 25, 26), 0.0, tuple(g.aabb_min), tuple(g.aabb_max))
    dc._its_sizes[key] = (1, 1)
    its = iso.get_intersection(g, compute_normals=True)
    assert all(_same(x, y) for x, y in zip((its.get_points(), its.get_normals(), its._cells, its._offsets),
                                           _reference_intersection(g, 0.0)))
    dc._dc_sizes[((24, 25, 26), 0.0, tuple(g.aabb_min), tuple(g.aabb_max))] = (1, 1)
    v, f = iso.dual_contouring(g, intersection=its)
    w, h = dc._dc_sequence(g, its, 1e-2, 1e-6)
    assert _same(v, w) and torch.equal(f, h)


# Points below the level in a corner, on an edge, on a face and inside the grid (one,
# two, four and eight active cells each): the last warp of the crossings full, short
# and of one cell.
@pytest.mark.parametrize("corner, edge, face, inner",
                         [(1, 0, 0, 0), (1, 1, 1, 3), (0, 0, 0, 4), (1, 0, 0, 4), (1, 1, 1, 7), (1, 0, 0, 8),
                          (0, 0, 0, 32), (1, 0, 0, 32)])
def test_few_cells(corner, edge, face, inner):
    vals = np.full((13, 12, 40), 1.0, np.float32)
    if corner:
        vals[0, 0, 0] = -0.3
    if edge:
        vals[0, 0, 20] = -0.2
    if face:
        vals[0, 6, 10] = -0.7
    at = [(x, y, z) for x in (3, 6, 9) for y in (3, 6, 9) for z in (3, 6, 9, 31, 34, 37)][:inner]
    for i, (x, y, z) in enumerate(at):
        vals[x, y, z] = -0.1 - 0.05 * i
    g = _grid(vals)
    its = iso.get_intersection(g, compute_normals=True)
    want = _reference_intersection(g, 0.0)
    assert its._cells.numel() == corner + 2 * edge + 4 * face + 8 * inner
    assert all(_same(x, y) for x, y in zip((its.get_points(), its.get_normals(), its._cells, its._offsets), want))
    assert _same(iso.get_intersection(g).get_points(), want[0])


def test_the_mesh_after_the_values_changed():
    """As many active cells elsewhere, the same cells with the signs swapped, and
    fewer cells: the mesh is the sequence's, bit for bit.  More cells than the
    intersection has dual vertices are refused."""
    vals = sphere((30, 31, 32), 0.5, center=(0.2, 0.0, 0.0))
    g = _grid(vals)
    for normals in (True, False):
        for other in (vals[::-1], -vals, sphere(vals.shape, 0.3)):
            g.set_values(torch.from_numpy(vals).cuda())
            its = iso.get_intersection(g, compute_normals=normals)
            g.set_values(torch.from_numpy(np.ascontiguousarray(other)).cuda())
            assert iso.get_intersection(g)._cells.numel() <= its._cells.numel()
            w, h = dc._dc_sequence(g, its, 1e-2, 1e-6)
            v, f = iso.dual_contouring(g, intersection=its)
            assert len(h) and _same(v, w) and torch.equal(f, h)
        g.set_values(torch.from_numpy(sphere(vals.shape, 0.7)).cuda())
        with pytest.raises(RuntimeError, match="more cells"):
            iso.dual_contouring(g, intersection=its)
