"""With the library's own allocations capped below any use, JumpFlood 2D on a
caller's workspace allocates nothing: a launch per pass, the oracle's deltas."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_jumpflood_2d_allocates_nothing(dol, O, cuda):
    torch = cuda
    L = dol.lib()
    dims = (200, 150)
    m = O.bool_to_mask(np.random.default_rng(1).random(dims[::-1]) < 0.02)
    start = O.border_init(m, dims)
    want = O.propagate("jumpflood", start, dims, 2)
    ws = torch.empty(L.dol_jumpflood_2d_workspace_size(*dims), dtype=torch.uint8, device="cuda")
    passes = {}
    for cap in (0, 1):
        L.dol_set_workspace_limit(C.c_size_t(cap))
        try:
            t = torch.from_numpy(start.copy()).cuda()
            names, ms = C.create_string_buffer(4096), (C.c_float * 64)()
            L.dol_profile_begin()
            dol.jumpflood(t, dims, 2, workspace=ws)
            n = L.dol_profile_end(names, C.c_size_t(4096), ms, 64)
            dol.sync()
        finally:
            L.dol_set_workspace_limit(C.c_size_t(0))
        np.testing.assert_array_equal(t.cpu().numpy(), want)
        passes[cap] = n
    assert passes[0] == 1    # the single launch, whose barrier needs a counter
    assert passes[1] == 8    # steps 128 .. 1
