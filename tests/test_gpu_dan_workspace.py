"""Danielsson's block engine on a caller's workspace at any 4-byte boundary: the
size that dol_danielsson_workspace_size gives is enough there, and nothing
outside it is written."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 4, 8, 12, 252])
@pytest.mark.parametrize("dims", [(200, 150), (300, 70), (90, 40, 21)])
def test_workspace_at_4_byte_boundaries(dol, O, cuda, dims, offset):
    torch = cuda
    L = dol.lib()
    rng = np.random.default_rng(sum(dims) + offset)
    m = O.bool_to_mask(rng.random(tuple(reversed(dims))) < 0.01)
    dl = dol.init_border(torch.from_numpy(m.view(np.int32)).cuda(), dims)
    d3 = dims if len(dims) == 3 else dims + (1,)
    need = L.dol_danielsson_workspace_size(*d3)
    assert need > 0
    buf = torch.full((need + 1024,), 0x5A, dtype=torch.uint8, device="cuda")
    fn = L.dol_danielsson_2d_ws if len(dims) == 2 else L.dol_danielsson_3d_ws
    dol.check(fn(*dims, C.c_void_p(dl.data_ptr()), 2, C.c_void_p(buf.data_ptr() + 256 + offset), C.c_size_t(need),
                 C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert L.dol_last_engine() == 1   # the blocks
    dol.sync()
    np.testing.assert_array_equal(dl.cpu().numpy(), O.propagate("danielsson", O.border_init(m, dims), dims, 2))
    b = buf.cpu().numpy()
    assert (b[:256 + offset] == 0x5A).all() and (b[256 + offset + need:] == 0x5A).all()
