"""Deltas to distances by row width: rows side by side in a warp (up to 32 cells),
parts of a row, several parts; with and without signs, cell widths 1, 2 and 3,
against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(w, h) for w in (1, 2, 3, 7, 10, 11, 16, 17, 31, 32, 33, 64, 65, 255, 257) for h in (1, 70)]
                         + [(w, 13, 41) for w in (1, 2, 3, 5, 11, 17, 30, 31, 33, 63, 65, 100, 129)])
def test_rows(dol, O, cuda, dims):
    rng = np.random.default_rng(sum(dims))
    dl = rng.integers(-600, 601, dims[::-1] + (len(dims),)).astype(np.int16)
    m = O.bool_to_mask(rng.random(dims[::-1]) < 0.5)
    t, md = cuda.from_numpy(dl).cuda(), cuda.from_numpy(m.view(np.int32)).cuda()
    for cw in (1, 2, 3):
        for sign, signd in ((None, None), (m, md)):
            got = dol.deltas_to_dist(t, dims, cw, sign_mask=signd)
            dol.sync()
            want = O.deltas_to_dist(dl, dims, cw, sign)
            np.testing.assert_array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32))
