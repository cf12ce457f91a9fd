"""The merge of coinciding vertices after marching cubes (mc_fix): a few merges in
a mesh of many tiles, tile edges, a position table of its own when the emit's
hash is full, levels hit by a whole plane of points, NaN values.  Checked against
the oracle's position weld, bit for bit."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from helpers import assert_same_mesh, noise, sphere  # noqa: E402


def _field(name):
    if name == "few":  # single points on the level in a mesh of ~200 tiles
        v = sphere((200, 200, 200), 0.77, center=(0.011, -0.017, 0.023))
        near = np.argwhere(np.abs(v) < 2e-3)
        for p in near[:: max(1, len(near) // 11)]:
            v[tuple(p)] = 0.0
        return v
    if name == "one_tile":  # V just below and faces just above one tile's rows
        v = sphere((34, 34, 34), 0.6)
        v[np.abs(v) < 4e-3] = 0.0
        return v
    if name == "plane":  # every point of a plane on the level, from both sides
        z = np.linspace(-1, 1, 65, dtype=np.float32)
        return np.ascontiguousarray(np.broadcast_to(np.where(z == 0, np.float32(0), np.float32(0.25) - np.abs(z)),
                                                    (70, 41, 65)).astype(np.float32))
    if name == "hash_full":  # more distinct positions than the emit's hash holds
        return noise((96, 96, 96), 5, 0.1)
    v = noise((40, 56, 48), 9, 0.2)  # "nan"
    v[np.random.default_rng(1).random(v.shape) < 0.02] = np.nan
    return v


@pytest.mark.parametrize("name,method", [("few", "nagae"), ("one_tile", "lorensen"), ("plane", "nagae"),
                                         ("hash_full", "lorensen")])
def test_merged_vertices_equal_the_oracle(oracle, name, method):
    import isoext_gb300 as iso

    vals = _field(name)
    grid = iso.UniformGrid(vals.shape)
    grid.set_values(torch.from_numpy(vals).cuda())
    v, f = iso.marching_cubes(grid, method=method)
    vo, fo, _ = oracle.mc_dense(vals, method=method)
    assert_same_mesh(v.cpu().numpy(), f.cpu().numpy(), vo, fo, name)


def test_merged_vertices_keep_their_edges():
    """iso_mc_dense_edges: each kept vertex's edge is one that it lies on."""
    from isoext_gb300 import diff

    vals = _field("few")
    x = torch.from_numpy(vals).cuda()
    v, f, e = diff._mc_forward(x, (-1.0,) * 3, (1.0,) * 3, 0.0, 0)
    n = torch.tensor(vals.shape, device="cuda")
    p, ax = e // 3, e % 3
    ijk = torch.stack([p // (n[1] * n[2]), (p // n[2]) % n[1], p % n[2]], -1)
    a = -1.0 + 2.0 * ijk.double() / (n - 1)
    h = 2.0 / (n - 1).double()
    off = v.double() - a
    along = off.gather(1, ax[:, None])[:, 0]
    across = off.scatter(1, ax[:, None], 0.0).abs().amax()
    assert float(across) < 1e-6 and float(along.min()) > -1e-6 and bool((along <= h[ax] + 1e-6).all())
    assert int(f.max()) == len(v) - 1 and len(torch.unique(f)) == len(v)


def test_nan_values_never_merge():
    """A vertex with a NaN coordinate equals no other; the rest of the mesh is
    merged as ever, and the call ends."""
    import isoext_gb300 as iso

    vals = _field("nan")
    grid = iso.UniformGrid(vals.shape)
    grid.set_values(torch.from_numpy(vals).cuda())
    v, f = iso.marching_cubes(grid)
    finite = torch.isfinite(v).all(-1)
    assert not bool(finite.all()) and int(f.max()) == len(v) - 1
    pos = v[finite]
    assert len(torch.unique(pos, dim=0)) == len(pos)
