"""The mask EDT around the line length below which a pass takes the plain form, in
either axis, and on lines too long for a staged tile: widths with and without
whole 16-byte rows, all three forms, with the workspace that the size function
gives and with the packed one.  Against the oracle's float envelope, beyond 4096
cells against the exact transform."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(37, 16), (37, 17), (40, 15), (900, 3), (3, 16384), (8, 13000), (13, 12600), (37, 16, 17), (37, 17, 16),
        (40, 16, 40), (41, 17, 17), (64, 3, 30), (65, 30, 3), (9, 2, 2), (250, 3, 90), (5, 300, 16)]


@pytest.mark.parametrize("dims", DIMS)
def test_short_and_long_lines(dol, O, cuda, dims):
    torch = cuda
    L = dol.lib()
    rng = np.random.default_rng(sum(dims))
    cells = int(np.prod(dims))
    size = L.dol_edt_mask_2d_workspace_size if len(dims) == 2 else L.dol_edt_mask_3d_workspace_size
    packed = (2 * cells + 255) // 256 * 256 + (4 * cells if len(dims) == 3 else 0)
    assert packed <= size(*dims)
    for p in (0.0, 0.002, 0.4):
        m = O.bool_to_mask(rng.random(tuple(reversed(dims))) < p)
        md = torch.from_numpy(m.view(np.int32)).cuda()
        if dims[1] > 4096:   # the reference's float envelope is not exact on such lines: the exact transform, transposed
            t = O.bool_to_mask(np.ascontiguousarray(O.mask_to_bool(m, dims).T))
            want = np.ascontiguousarray(O.sdf_signed_exact_thin(t, dims[::-1]).T)
        else:
            want = np.asarray(O.sdf_signed_felzenszwalb(m, dims), np.float32)
        sq = None
        for n in (size(*dims), packed):
            ws = torch.empty(n, dtype=torch.uint8, device="cuda")
            got = dol.edt_mask(md, dims, dol.EDT_SIGNED, workspace=ws).cpu().numpy()
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), p
            forms = [dol.edt_mask(md, dims, f, workspace=ws).cpu().numpy() for f in (dol.EDT_SQUARED, dol.EDT_DIST)]
            if sq is not None:
                assert all(np.array_equal(a, b) for a, b in zip(sq, forms))
            sq = forms
