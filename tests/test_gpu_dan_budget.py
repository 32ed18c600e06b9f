"""Danielsson on deltas that the block iteration does not settle within its budget
of rounds, so that the serial walk takes a phase over: the oracle's deltas, no
timeout, on images and volumes of every row shape of the walk, on a caller's
workspace as well."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = 8   # DOL_TUNE_DANIELSSON_ROWS


@pytest.mark.parametrize("dims", [(50, 700), (100, 300), (200, 150), (400, 120), (700, 90), (1500, 70), (60, 40, 12),
                                  (120, 30, 14), (250, 24, 12), (300, 20, 12), (600, 16, 10), (1100, 12, 8)])
def test_budget_runs_out(dol, O, cuda, dims):
    torch = cuda
    L = dol.lib()
    rng = np.random.default_rng(sum(dims))
    shape = dims[::-1] + (len(dims),)
    far = 8192 if len(dims) == 2 else 25000
    fields = [rng.integers(-2000, 2001, shape), rng.integers(-32768, 32768, shape),
              np.where(rng.random(shape[:-1] + (1,)) < 0.02, rng.integers(-300, 301, shape), far)]
    d3 = dims if len(dims) == 3 else dims + (1,)
    L.dol_tune_set(ROWS, dims[0], 4)   # the blocks, whatever the shape
    try:
        need = L.dol_danielsson_workspace_size(*d3)
        for i, f in enumerate(fields):
            f = f.astype(np.int16)
            want = O.propagate("danielsson", f, dims, 2)
            t = torch.from_numpy(f.copy()).cuda()
            dol.danielsson(t, dims, 2)
            assert L.dol_last_engine() == 1
            dol.sync()
            np.testing.assert_array_equal(t.cpu().numpy(), want, err_msg=f"field {i}")
            t = torch.from_numpy(f.copy()).cuda()
            ws = torch.empty(need, dtype=torch.uint8, device="cuda")
            fn = L.dol_danielsson_2d_ws if len(dims) == 2 else L.dol_danielsson_3d_ws
            dol.check(fn(*dims, C.c_void_p(t.data_ptr()), 2, C.c_void_p(ws.data_ptr()), C.c_size_t(need),
                         C.c_void_p(torch.cuda.current_stream().cuda_stream)))
            dol.sync()
            np.testing.assert_array_equal(t.cpu().numpy(), want, err_msg=f"field {i}")
    finally:
        L.dol_tune_set(ROWS, dims[0], 0)
