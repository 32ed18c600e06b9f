"""The mask EDT at widths that are no multiple of 8 (padded intermediate rows),
in tiles shared by several CTAs, with lines too long for 16-column tiles, and
on scratch that only holds packed rows: the oracle's floats bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mask(O, dims, p):
    rng = np.random.default_rng(sum(dims) + int(1000 * p))
    return O.bool_to_mask(rng.random(tuple(reversed(dims))) < p)


@pytest.mark.parametrize("dims", [(1, 5), (7, 300), (9, 65), (31, 257), (1501, 130), (33, 2900), (21, 3100), (40, 4000),
                                  (1, 3, 4), (9, 12, 10), (33, 70, 300), (129, 31, 65)])
@pytest.mark.parametrize("p", [0.5, 0.02, 0.0005])
def test_odd_widths_match_oracle(dol, O, cuda, dims, p):
    m = _mask(O, dims, p)
    md = cuda.from_numpy(m.view(np.int32)).cuda()
    want = np.asarray(O.sdf_signed_felzenszwalb(m, dims), np.float32).view(np.uint32)
    assert np.array_equal(dol.edt_mask(md, dims, dol.EDT_SIGNED).cpu().numpy().view(np.uint32), want)
    # scratch for packed rows only: the size before rows were padded
    cells = int(np.prod(dims))
    packed = (2 * cells + 255) // 256 * 256 + (4 * cells if len(dims) == 3 else 0)
    if len(dims) == 2:
        packed = (2 * cells + 255) // 256 * 256
    ws = cuda.empty(packed, dtype=cuda.uint8, device="cuda")
    out = dol.edt_mask(md, dims, dol.EDT_SIGNED, workspace=ws)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
    L = dol.lib()
    try:   # and a cap on the library's own scratch between the two sizes
        L.dol_set_workspace_limit(C.c_size_t(packed))
        out = dol.edt_mask(md, dims, dol.EDT_SIGNED)
    finally:
        L.dol_set_workspace_limit(C.c_size_t(0))
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
