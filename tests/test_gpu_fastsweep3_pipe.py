"""FastSweep 3D's streaming columns: the oracle's deltas at the edges of the
kernel's ranges (columns that are full or ragged, part of a chunk of slices, one
more than the ring holds, more columns than stay resident), on sparse, dense and
empty masks, and on scratch too small for it."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 2, 2), (5, 40, 3), (64, 9, 5), (65, 33, 6), (128, 20, 9), (129, 31, 14),
                                  (256, 12, 10), (257, 12, 10), (31, 3, 70), (40, 70, 41),
                                  (16, 16, 57), (33, 17, 64), (17, 40, 130), (300, 18, 9), (100, 100, 17)])
@pytest.mark.parametrize("p", [0.0, 0.003, 0.3])
def test_columns_match_oracle(dol, O, cuda, dims, p):
    rng = np.random.default_rng(sum(dims) + int(1000 * p))
    m = O.bool_to_mask(rng.random((dims[2], dims[1], dims[0])) < p)
    md = cuda.from_numpy(m.view(np.int32)).cuda()
    for cw, init in ((2, O.border_init), (1, O.init_deltas)):
        base = init(m, dims)
        want = O.propagate("fastsweep", base.copy(), dims, cw)
        got = dol.fastsweep(cuda.from_numpy(base.copy()).cuda(), dims, cw)
        dol.sync()
        np.testing.assert_array_equal(got.cpu().numpy(), want)
    # scratch of the row engines only: the size before this kernel
    rows = (4 * dims[1] * dims[2] + 255) // 256 * 256 + (4 * (dims[1] + dims[2] + 2) + 255) // 256 * 256 + 256
    ws = cuda.empty(rows, dtype=cuda.uint8, device="cuda")
    got = dol.fastsweep(cuda.from_numpy(base.copy()).cuda(), dims, cw, workspace=ws)
    dol.sync()
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    L = dol.lib()
    try:
        L.dol_set_workspace_limit(C.c_size_t(rows))
        got = dol.fastsweep(cuda.from_numpy(base.copy()).cuda(), dims, cw)
        dol.sync()
    finally:
        L.dol_set_workspace_limit(C.c_size_t(0))
    np.testing.assert_array_equal(got.cpu().numpy(), want)


def test_arbitrary_deltas(dol, O, cuda):
    """Any int16 components, so that shifts wrap: still the oracle's deltas."""
    rng = np.random.default_rng(9)
    dims = (70, 33, 21)
    base = rng.integers(-32768, 32768, size=(dims[2], dims[1], dims[0], 3)).astype(np.int16)
    want = O.propagate("fastsweep", base.copy(), dims, 2)
    got = dol.fastsweep(cuda.from_numpy(base.copy()).cuda(), dims, 2)
    dol.sync()
    np.testing.assert_array_equal(got.cpu().numpy(), want)
