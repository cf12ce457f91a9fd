"""Dual contouring on boxes whose grid coordinates repeat: the weld through a table
against the call sequence's hash weld, bit for bit, on grids where a search of the
cells that share a coordinate would be quadratic (a box of no extent: every
vertex lies in every cell), and the rule that tells such boxes."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

import isoext_gb300 as iso  # noqa: E402
from helpers import noise, sphere  # noqa: E402
from isoext_gb300 import _ffi, dc, diff  # noqa: E402
from isoext_gb300.grids import grid_positions  # noqa: E402

BOXES = {
    "point": ((0.5,) * 3, (0.5,) * 3),
    "plane": ((-1.0, -1.0, 2.0), (1.0, 1.0, 2.0)),
    "line": ((-1.0, 3.0, 2.0), (1.0, 3.0, 2.0)),
    "far": ((1e6,) * 3, (1e6 + 1,) * 3),
    "far_x": ((1e6, -1.0, -1.0), (1e6 + 2, 1.0, 1.0)),
    "reversed": ((1e6 + 3, 1.0, -1.0), (1e6, -1.0, 1.0)),
    "zero": ((0.0,) * 3, (0.0,) * 3),
}


def _same(a, b):
    return (a is None) == (b is None) and (a is None or torch.equal(a.view(torch.int32), b.view(torch.int32)))


def _values(kind):
    if kind == "sphere":
        return sphere((128, 120, 136), 0.7, center=(0.02, -0.01, 0.03))
    return noise((37, 41, 39), 3, 0.1)


@pytest.mark.parametrize("kind", ["sphere", "noise"])
@pytest.mark.parametrize("box", list(BOXES))
def test_sparse(box, kind):
    vals = _values(kind)
    nx, ny, nz = vals.shape
    v = torch.from_numpy(vals).cuda()
    corners = torch.stack([v[i:nx - 1 + i, j:ny - 1 + j, k:nz - 1 + k] for i in (0, 1) for j in (0, 1) for k in (0, 1)],
                          -1).reshape(-1, 8)
    g = iso.SparseGrid(vals.shape, *BOXES[box])
    g.add_cells(torch.arange(len(corners), dtype=torch.int32, device="cuda"))
    g.set_values(corners)
    a, f = iso.dual_contouring(g)
    b, h = iso.dual_contouring(g, intersection=iso.get_intersection(g, compute_normals=True))
    assert f.numel() and _same(a, b) and torch.equal(f, h)


@pytest.mark.parametrize("kind", ["sphere", "noise"])
@pytest.mark.parametrize("box", list(BOXES))
def test_dense(box, kind):
    """The call without an intersection and the one with it against the sequence;
    the differentiable one has the same mesh."""
    vals = _values(kind)
    g = iso.UniformGrid(vals.shape, *BOXES[box])
    g.set_values(torch.from_numpy(vals).cuda())
    its = iso.get_intersection(g, compute_normals=True)
    b, h = dc._dc_sequence(g, its, 1e-2, 1e-6)
    for a, f in (iso.dual_contouring(g), iso.dual_contouring(g, intersection=its),
                 diff.dual_contouring(g.get_values(), *BOXES[box])):
        assert f.numel() and _same(a, b) and torch.equal(f, h)


# In a captured graph, replayed on other values, and with the vertices 4 bytes off
# the 8-byte boundary that the entries (then the table) need: the room for the list
# of vertices on faces is one short, and on these boxes every vertex lies on one.
# "mirrored" has distinct coordinates: the local search over all cells.
@pytest.mark.parametrize("box", ["point", "reversed", "mirrored"])
def test_capture_and_a_full_face_list(box):
    lo, hi = BOXES.get(box, ((1.0,) * 3, (-1.0,) * 3))
    lib = _ffi.lib()
    fields = [torch.from_numpy(noise((21, 22, 35), seed, 0.1)).cuda() for seed in (1, 2)]
    want = []
    for x in fields:
        g = iso.UniformGrid(x.shape, lo, hi)
        g.set_values(x)
        its = iso.get_intersection(g, compute_normals=True)
        want.append((*dc._dc_sequence(g, its, 1e-2, 1e-6), its._cells.numel()))
    values = fields[0].clone()
    for capA, offset in ((want[0][2], 1), (1 << 15, 0)):
        ws = torch.empty(dc.dc_workspace_bytes(values.shape, capA, 1 << 17), dtype=torch.uint8, device="cuda")
        vout = torch.empty(3 * capA + offset, device="cuda")[offset:]
        fout = torch.empty((1 << 17, 3), dtype=torch.int32, device="cuda")
        small = torch.zeros(8, dtype=torch.int64, device="cuda")
        assert vout.data_ptr() % 8 == 4 * offset

        def call():
            small.zero_()
            _ffi.check(dc.dc_dense_into(values, lo, hi, 0.0, 1e-2, 1e-6, vout.view(-1, 3), fout, ws, small,
                                        torch.cuda.current_stream().cuda_stream))

        def check(k):
            V, F, status = int(small[0]), int(small[1]), int(small[6]) & 0xffffffff
            assert status == 0 and V == len(want[k][0]) and F == len(want[k][1])
            assert _same(vout[:3 * V].view(-1, 3), want[k][0]) and torch.equal(fout[:F], want[k][1])

        values.copy_(fields[0])
        call()
        check(0)
        if offset:
            continue
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            call()
        for k in (1, 0):
            values.copy_(fields[k])
            graph.replay()
            torch.cuda.synchronize()
            check(k)


# Spacings just above the rule's line, 2^-20 of the box's magnitude: no coordinate repeats.
@pytest.mark.parametrize("arith", ["nvcc", "host"])
def test_coordinates_above_the_line_are_distinct(arith):
    iso.set_arithmetic(arith)
    try:
        rng = np.random.default_rng(0)
        for n in (2, 3, 17, 129, 1000, 4097, 1 << 20):
            index = torch.arange(n, device="cuda")
            for _ in range(8):
                lo = float(np.float32(rng.choice([-1, 1]) * 2.0 ** rng.uniform(-20, 20)))
                # h = 2^-20 max(|lo|, |lo + (n - 1) h|), a little above
                h = abs(lo) * 2.0 ** -20 * 1.0005
                if lo > 0:
                    h /= max(1 - (n - 1) * 2.0 ** -20, 2.0 ** -20)
                x = grid_positions(index, n, lo, float(np.float32(lo + h * (n - 1))))
                assert bool((x[1:] > x[:-1]).all()), (n, lo)
    finally:
        iso.set_arithmetic("nvcc")
