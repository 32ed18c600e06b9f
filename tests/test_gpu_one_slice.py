"""Volumes of one slice through the 3D entries that keep no deltas of the
caller's: 3D cells and their scratch fit the workspace that the size functions
give, nothing outside it is written, and the distances are the oracle's."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
METHODS = ["danielsson", "fastsweep", "jumpflood"]


@pytest.mark.parametrize("w,h", [(40, 40), (70, 33), (5, 3)])
@pytest.mark.parametrize("method", METHODS)
def test_one_slice(dol, O, cuda, method, w, h):
    torch = cuda
    L = dol.lib()
    dims = (w, h, 1)
    rng = np.random.default_rng(w + h)
    m = O.bool_to_mask(rng.random((1, h, w)) < 0.1)
    md = torch.from_numpy(m.view(np.int32)).cuda()
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    num = dol.METHODS[method]
    ptr = lambda t: C.c_void_p(t.data_ptr())
    dist = torch.empty(dims[::-1], dtype=torch.float32, device="cuda")
    for two_pass in (False, True):
        size = L.dol_sdf_two_pass_workspace_size if two_pass else L.dol_sdf_workspace_size
        need = size(w, h, 1, num)
        buf = torch.full((need + 512 + 32 * w * h,), 0x5A, dtype=torch.uint8, device="cuda")
        work = C.c_void_p(buf.data_ptr() + 256)
        if two_pass:
            dol.check(L.dol_sdf_two_pass_3d(w, h, 1, ptr(md), num, None, None, ptr(dist), work, C.c_size_t(need), stream))
            ext, intr = (O.deltas_to_dist(O.propagate(method, O.init_deltas(m, dims, inv), dims, 1), dims, 1)
                         for inv in (False, True))
            want = ext - intr
        else:
            dol.check(L.dol_sdf_3d(w, h, 1, ptr(md), num, None, ptr(dist), work, C.c_size_t(need), stream))
            want = O.deltas_to_dist(O.propagate(method, O.border_init(m, dims), dims, 2), dims, 2, m)
        dol.sync()
        np.testing.assert_array_equal(dist.cpu().numpy().reshape(want.shape), want)
        b = buf.cpu().numpy()
        assert (b[:256] == 0x5A).all() and (b[256 + need:] == 0x5A).all()


@pytest.mark.parametrize("method", METHODS)
def test_the_2d_entry_still_takes_its_own_size(dol, O, cuda, method):
    """what the 2D entry needs is no more than before the size covered both"""
    torch = cuda
    L = dol.lib()
    w, h = 200, 300
    m = O.bool_to_mask(np.random.default_rng(3).random((h, w)) < 0.05)
    md = torch.from_numpy(m.view(np.int32)).cuda()
    up = lambda b: (b + 255) // 256 * 256
    need = up(4 * w * h)
    if method == "jumpflood":
        need += up(L.dol_jumpflood_2d_workspace_size(w, h))
    if method == "danielsson":
        need += up(L.dol_danielsson_workspace_size(w, h, 1))
    assert need <= L.dol_sdf_workspace_size(w, h, 1, dol.METHODS[method])
    work = torch.empty(need, dtype=torch.uint8, device="cuda")
    _, dist = dol.sdf(md, (w, h), method, want_deltas=False, workspace=work)
    dol.sync()
    dims = (w, h)
    want = O.deltas_to_dist(O.propagate(method, O.border_init(m, dims), dims, 2), dims, 2, m)
    np.testing.assert_array_equal(dist.cpu().numpy(), want)
