"""Every cell active, with more face indices (6 per quad) than 31 bits count and
crossings that still fit: the intersection has no faces, and neither the two-step
flow nor the sparse one bounds them.  About 45 GB of device memory."""

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

import isoext_gb300 as iso  # noqa: E402

N = 494


def test_more_face_indices_than_31_bits():
    if torch.cuda.mem_get_info()[0] < 100 << 30:
        pytest.skip("needs 100 GB of free device memory")
    A, Q = (N - 1) ** 3, 3 * (N - 2) ** 2 * (N - 1)
    assert 6 * Q >= 1 << 31 and 12 * A < 1 << 31
    i = torch.arange(N, device="cuda")
    odd = ((i[:, None, None] + i[None, :, None] + i[None, None, :]) & 1).bool()  # a checkerboard
    g = iso.UniformGrid([N] * 3)
    g.set_values(torch.where(odd, 1.0, -1.0))
    del odd
    its = iso.get_intersection(g)
    assert its.get_points().shape == (12 * A, 3)
    assert its._cells.numel() == A and int(its._offsets[-1]) == 12 * A
    assert torch.equal(its._cells[-1000:].cpu(), torch.arange(A - 1000, A, dtype=torch.int32))
    v, f = iso.dual_contouring(g, 0.0, its)
    assert v.shape == (A, 3) and f.shape == (2 * Q, 3)
    del its, g
    torch.cuda.empty_cache()
    # the same cells in a sparse grid: the same mesh
    s = iso.SparseGrid([N] * 3)
    ids = torch.arange(A, dtype=torch.int32, device="cuda")
    s.add_cells(ids)
    m = N - 1
    par = (ids // (m * m) + ids // m % m + ids % m) & 1
    corner = torch.tensor([0, 1, 1, 0, 1, 0, 0, 1], device="cuda")  # parity of 4x + 2y + z
    for k in range(8):
        s._values[:, k] = torch.where(((par + corner[k]) & 1).bool(), 1.0, -1.0)
    del ids, par
    vs, fs = iso.dual_contouring(s)
    assert torch.equal(vs, v) and torch.equal(fs, f)
    del s, vs, fs, f, v
    torch.cuda.empty_cache()
