"""Danielsson and FastSweep on both sides of the lines at which another engine
takes over (rows that fill a warp or do not, few wide rows, one row per slice,
short chains, thin volumes), against the oracle: mask fields and deltas that a
caller brings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

IMAGES = [(1, 40), (31, 33), (32, 33), (33, 40), (63, 30), (64, 40), (65, 29), (111, 31), (112, 33), (255, 33),
          (257, 23), (257, 24), (512, 31), (513, 31), (513, 32), (1024, 12), (1025, 9), (2048, 31), (2049, 30),
          (2049, 127), (2049, 128), (4096, 3)]
VOLUMES = [(1, 1, 40), (3, 5, 7), (32, 6, 9), (33, 8, 5), (64, 1, 30), (65, 9, 4), (127, 5, 6), (129, 7, 3), (255, 4, 5),
           (256, 1, 9), (256, 5, 5), (257, 3, 5), (513, 4, 3), (1025, 2, 3), (1199, 2, 3), (1200, 2, 3), (2049, 3, 3),
           (20, 3, 34), (64, 40, 17), (64, 40, 18), (40, 60, 3)]


@pytest.mark.parametrize("dims", IMAGES + VOLUMES)
def test_engines(dol, O, cuda, dims):
    rng = np.random.default_rng(sum(dims) * 3 + len(dims))
    methods = ["danielsson"] + (["fastsweep"] if len(dims) == 2 or dims[0] <= 2048 else [])
    fields = []
    for p in (0.004, 0.2):
        m = O.bool_to_mask(rng.random(tuple(reversed(dims))) < p)
        fields += [(O.border_init(m, dims), 2), (O.init_deltas(m, dims), 1)]
    f = rng.integers(-300, 301, fields[0][0].shape).astype(np.int16)
    f[rng.random(f.shape[:-1]) < 0.8] = 8192 if len(dims) == 2 else 25000
    fields.append((f, 3))
    for i, (f, cw) in enumerate(fields):
        for method in methods:
            got = dol.propagate(method, cuda.from_numpy(f.copy()).cuda(), dims, cw)
            dol.sync()
            np.testing.assert_array_equal(got.cpu().numpy(), O.propagate(method, f, dims, cw),
                                          err_msg=f"{method} field {i}")
