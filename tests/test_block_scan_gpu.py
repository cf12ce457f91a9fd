"""The scan of block sums over the rounds of its one CTA (4096 sums each) and
with block sums on and off 16-byte boundaries, through the sparse grid's filter
(a sum per 256 cells): the kept ids in order, exactly."""

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from isoext_gb300 import _ffi  # noqa: E402
from isoext_gb300.sparse import _p, _stream  # noqa: E402


@pytest.mark.parametrize("offset", [0, 8])
@pytest.mark.parametrize("blocks", [1, 33, 1024, 4095, 4096, 4097, 9000])
def test_filter_over_scan_rounds(blocks, offset):
    m = blocks * 256 - (blocks > 1) * 17
    g = np.random.default_rng([blocks, offset])
    keep = g.random(m) < 0.3
    vals = torch.ones((m, 8), dtype=torch.float32, device="cuda")
    vals[:, 3] = torch.from_numpy(np.where(keep, -1.0, 1.0).astype(np.float32)).cuda()
    ids = torch.arange(m, dtype=torch.int32, device="cuda") * 3
    lib = _ffi.lib()
    blk = torch.zeros(int(lib.iso_sparse_blocks_size(m)) // 8 + 2, dtype=torch.int64, device="cuda")
    counts = torch.zeros(2, dtype=torch.int64, device="cuda")
    st, at = _stream(torch.device("cuda")), C.c_void_p(blk.data_ptr() + offset)
    _ffi.check(lib.iso_sparse_filter_count(_p(vals), m, 0.0, at, _p(counts), st))
    assert counts.cpu().tolist() == [int(keep.sum()), 0]
    out = torch.empty(int(keep.sum()), dtype=torch.int32, device="cuda")
    _ffi.check(lib.iso_sparse_filter_write(_p(ids), _p(vals), m, 0.0, at, _p(out), st))
    assert np.array_equal(out.cpu().numpy(), np.flatnonzero(keep).astype(np.int32) * 3)
