"""Float Felzenszwalb where boundaries nearly tie: heights whose parabolas lie on
a line or on a slightly bent curve but for 2^-18 to 2^-25 of a boundary's size,
so that rounding decides which stay.  The oracle's floats, bit for bit; and
input that is not finite ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 333, 1024])
@pytest.mark.parametrize("bend", [0.0, 1e-7, 3e-6, 1e-4])
def test_near_ties(dol, O, cuda, n, bend):
    rng = np.random.default_rng(int(bend * 1e8) + n)
    for shape in ((n, 64), (64, n)):
        line = 0 if shape[0] == n else 1
        q = np.arange(n, dtype=np.float64)
        q = q[:, None] if line == 0 else q[None, :]
        for _ in range(6):
            slope = rng.uniform(-3, 3) * n
            size = np.abs(slope) + n
            rough = 2.0 ** rng.uniform(-25, -18, shape) * size * rng.uniform(-1, 1, shape)
            runs = np.where(rng.random(shape) < 0.1, rng.uniform(0, 40, shape), 0.0)   # some far above
            f = (rng.uniform(0, 1000) + slope * q + bend * size * (q - n / 2) ** 2 / n - q * q + rough + runs)
            f = f.astype(np.float32)
            dims = (shape[1], shape[0])
            want = np.asarray(O.felzenszwalb(f, dims), np.float32)
            got = dol.felzenszwalb(cuda.from_numpy(f.copy()).cuda(), dims).cpu().numpy()
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


def test_not_finite_ends(dol, O, cuda):
    rng = np.random.default_rng(1)
    dims = (70, 90)
    good = (100 * rng.random((90, 70))).astype(np.float32)
    for bad in (np.inf, -np.inf, np.nan):
        for share in (0.01, 0.5, 1.0):
            f = np.where(rng.random(good.shape) < share, np.float32(bad), good)
            dol.felzenszwalb(cuda.from_numpy(f).cuda(), dims)
            dol.sync()
    got = dol.felzenszwalb(cuda.from_numpy(good.copy()).cuda(), dims).cpu().numpy()
    assert np.array_equal(got, np.asarray(O.felzenszwalb(good, dims), np.float32))
