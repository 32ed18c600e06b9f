"""JumpFlood 3D on deltas that the packed sites cannot hold, at sizes where the
passes that take over change their run of slices and span many CTAs: the
oracle's deltas."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 2, 3), (33, 9, 70), (70, 40, 33), (80, 82, 80), (40, 300, 50), (128, 129, 130)])
@pytest.mark.parametrize("kind", ["arbitrary", "one_far"])
def test_passes_on_cells(dol, O, cuda, dims, kind):
    rng = np.random.default_rng(sum(dims))
    if kind == "arbitrary":
        f = rng.integers(-400, 401, dims[::-1] + (3,)).astype(np.int16)
        f[rng.random(dims[::-1]) < 0.7] = 25000
        f[0, 0, 0] = (-30000, 2, 1)
    else:
        m = O.bool_to_mask(rng.random(dims[::-1]) < 0.05)
        f = O.border_init(m, dims)
        f[-1, -1, -1] = (3, -1500, 5)
    got = dol.jumpflood(cuda.from_numpy(f.copy()).cuda(), dims, 2)
    dol.sync()
    np.testing.assert_array_equal(got.cpu().numpy(), O.propagate("jumpflood", f, dims, 2))
