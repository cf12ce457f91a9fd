"""The union grid where its paths change: rows, and tiles of 32 z by 4 y by 4 x
from 2^21 points on, both over widths that fill them or not; unions of up to 32
primitives, far and touching ones, boxes of very small and very large
coordinates, parameters that are negative, infinite or NaN.  Every point exactly
against the formula over all primitives: leaving a primitive out of a tile
must never show."""

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from isoext_gb300 import UniformGrid, _ffi  # noqa: E402
from isoext_gb300.serve import prims_buffer  # noqa: E402


def _prims(g, k, scale, reach):
    p = np.zeros((k, 7), np.float32)
    p[:, 0] = g.integers(0, 2, k)
    p[:, 1:4] = g.uniform(-reach, reach, (k, 3)) * scale
    p[:, 4:7] = g.uniform(0.02, 0.4, (k, 3)) * scale
    return p


def _union(points, prims):
    """The formulas in FP32, a NaN distance passed over as fminf passes it."""
    f = np.float32
    d = np.full(points.shape[:-1], np.finfo(np.float32).max, np.float32)
    for row in prims:
        dx, dy, dz = (points[..., k] - row[1 + k] for k in range(3))
        if row[0] == 0:
            dk = np.sqrt((dx * dx + dy * dy) + dz * dz) - row[4]
        else:
            qx, qy, qz = np.abs(dx) - row[4], np.abs(dy) - row[5], np.abs(dz) - row[6]
            ox, oy, oz = (np.fmax(q, f(0)) for q in (qx, qy, qz))
            dk = np.sqrt((ox * ox + oy * oy) + oz * oz) + np.fmin(np.fmax(np.fmax(qx, qy), qz), f(0))
        d = np.fmin(d, dk)
    assert d.dtype == np.float32
    return d


def _check(shape, lo, hi, prims):
    grid = UniformGrid(list(shape), lo, hi)
    dev = torch.from_numpy(prims_buffer(prims)).cuda()
    _ffi.check(_ffi.lib().iso_sdf_union_grid(C.c_void_p(dev.data_ptr()), *shape, _ffi.fvec3(lo), _ffi.fvec3(hi),
                                             C.c_void_p(grid._values.data_ptr()),
                                             C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    got = grid.get_values().cpu().numpy()
    with np.errstate(all="ignore"):
        want = _union(grid.get_points().cpu().numpy(), prims)
    assert np.array_equal(got, want)  # no NaN on either side


@pytest.mark.parametrize("shape", [(5, 7, 33), (127, 129, 128), (128, 128, 128), (129, 128, 131), (1, 1025, 2050),
                                   (700, 3, 1000), (700, 4, 800), (400, 400, 16), (400, 400, 17), (4000, 31, 17)])
@pytest.mark.parametrize("k", [1, 10, 32])
def test_shapes(shape, k):
    g = np.random.default_rng([*shape, k])
    _check(shape, (-1, -1, -1), (1, 1, 1), _prims(g, k, 1.0, 0.9))


@pytest.mark.parametrize("scale", [1e-24, 1e-12, 1e-3, 1e4, 1e15, 3e18, 1e25])
def test_scales(scale):
    g = np.random.default_rng(int(abs(np.log2(scale))))
    _check((129, 126, 130), (-scale, -0.3 * scale, 0.1 * scale), (scale, scale, 2 * scale), _prims(g, 20, scale, 3.0))


@pytest.mark.parametrize("case", ["lattice", "negative", "same", "inf", "nan", "huge"])
def test_special_primitives(case):
    g = np.random.default_rng(3)
    p = _prims(g, 12, 1.0, 0.8)
    if case == "lattice":  # equal distances, exactly
        p[:, 1:] = np.round(p[:, 1:] * 8) / 8
    elif case == "negative":
        p[::2, 4:] *= -1
    elif case == "same":
        p[6:] = p[:6]
    elif case == "inf":
        p[0, 4], p[3, 1], p[5, 2] = -np.inf, np.inf, -np.inf
    elif case == "nan":
        p[1, 4], p[7, 2] = np.nan, np.nan
    elif case == "huge":
        p[2, 1], p[4, 4], p[9, 3] = 1e30, -1e20, -5e18
    _check((130, 128, 129), (-1, -1, -1), (1, 1, 1), p)
