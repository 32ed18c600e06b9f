"""The 3D in-place occlusion sweep's pipelined blocks: the oracle's floats bit for
bit where blocks, lanes and rows are ragged, on aligned and unaligned rows, on
fields that are not 0 / 1, and with no scratch allowed."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (1, 40, 3), (31, 17, 33), (32, 16, 32), (33, 16, 32), (64, 15, 65),
                                  (36, 50, 9), (100, 3, 70), (7, 90, 90), (130, 35, 34),
                                  (32, 16, 48), (33, 17, 49), (5, 16, 97)])
@pytest.mark.parametrize("kind", ["mask", "weights"])
def test_wave_matches_oracle(dol, O, cuda, dims, kind):
    rng = np.random.default_rng(sum(dims))
    w, h, d = dims
    f = np.empty((8, d, h, w), np.float32)
    if kind == "mask":
        f[:] = (rng.random((d, h, w)) < 0.1).astype(np.float32)
    else:
        f[:] = rng.random(f.shape)
    want = O.occlusion_sweep(f.copy(), dims)
    got = dol.occlusion_sweep(cuda.from_numpy(f.copy()).cuda(), dims).cpu().numpy()
    assert np.array_equal(got.view(np.uint32), np.asarray(want, np.float32).view(np.uint32))
    L = dol.lib()
    try:
        L.dol_set_workspace_limit(C.c_size_t(1))
        got = dol.occlusion_sweep(cuda.from_numpy(f.copy()).cuda(), dims).cpu().numpy()
    finally:
        L.dol_set_workspace_limit(C.c_size_t(0))
    assert np.array_equal(got.view(np.uint32), np.asarray(want, np.float32).view(np.uint32))
