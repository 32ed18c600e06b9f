"""JumpFlood 3D on packed sites: the oracle's deltas at the last sides that fit
the packing and the first that do not, on ragged and degenerate shapes, and on
deltas that it cannot hold (arbitrary values, cells partly at max), which the
general passes take over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 2), (2, 1, 1), (5, 3, 2), (33, 9, 70), (6, 4, 8), (7, 5, 17), (128, 130, 67), (64, 32, 16), (300, 5, 4), (4, 301, 5),
                                  (6, 4, 598), (600, 3, 2), (37, 41, 43)])
@pytest.mark.parametrize("p", [0.0, 0.002, 0.4])
def test_packed_matches_oracle(dol, O, cuda, dims, p):
    rng = np.random.default_rng(sum(dims) + int(1000 * p))
    m = O.bool_to_mask(rng.random((dims[2], dims[1], dims[0])) < p)
    md = cuda.from_numpy(m.view(np.int32)).cuda()
    for cw, init in ((2, O.border_init), (1, O.init_deltas)):
        want = O.propagate("jumpflood", init(m, dims).copy(), dims, cw)
        got = dol.jumpflood(cuda.from_numpy(init(m, dims)).cuda(), dims, cw)
        dol.sync()
        np.testing.assert_array_equal(got.cpu().numpy(), want)
    dl, _ = dol.sdf(md, dims, "jumpflood")
    np.testing.assert_array_equal(dl.cpu().numpy(), O.propagate("jumpflood", O.border_init(m, dims), dims, 2))


@pytest.mark.parametrize("dims", [(16, 16, 16), (19, 6, 11)])
@pytest.mark.parametrize("kind", ["arbitrary", "part_max", "one_far"])
def test_deltas_that_do_not_pack(dol, O, cuda, dims, kind):
    rng = np.random.default_rng(sum(dims))
    shape = (dims[2], dims[1], dims[0], 3)
    if kind == "arbitrary":
        f = rng.integers(-32768, 32768, size=shape).astype(np.int16)
    else:
        f = np.full(shape, 25000, np.int16)
        f[rng.random(shape[:3]) < 0.1] = 0
        if kind == "part_max":
            f[1, 2, 3] = (25000, 0, 0)
            f[2, 1, 1] = (1, 25000, 2)
        else:
            f[-1, -1, -1] = (3, -700, 5)
    want = O.propagate("jumpflood", f.copy(), dims, 2)
    got = dol.jumpflood(cuda.from_numpy(f.copy()).cuda(), dims, 2)
    dol.sync()
    np.testing.assert_array_equal(got.cpu().numpy(), want)
