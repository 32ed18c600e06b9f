"""Chamfer in blocks of 32 rows: whole numbers equal to the oracle's at the
edges of blocks, warps and threads, on scattered seeds, arbitrary values and
fields whose only seed sits in one corner (carried through every block)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2, 64), (5, 97), (127, 63), (128, 64), (129, 65), (257, 96), (1025, 130), (4096, 70),
                                  (33, 1000)])
@pytest.mark.parametrize("dtype", [np.int16, np.int32])
def test_blocks_match_oracle(dol, O, cuda, dims, dtype):
    rng = np.random.default_rng(sum(dims))
    shape = (dims[1], dims[0])
    top = np.iinfo(dtype).max - 16
    fields = [rng.integers(np.iinfo(dtype).min, np.iinfo(dtype).max - 4, size=shape, endpoint=True).astype(dtype),
              np.where(rng.random(shape) < 0.003, 0, top).astype(dtype)]
    for y, x in ((0, 0), (0, -1), (-1, 0), (-1, -1), (shape[0] // 2, shape[1] // 2)):
        f = np.full(shape, top, dtype)
        f[y, x] = 0
        fields.append(f)
    for i, f in enumerate(fields):
        t = cuda.from_numpy(f.copy()).cuda()
        assert dol.chamfer(t, dims) == 3
        np.testing.assert_array_equal(t.cpu().numpy(), O.chamfer(f, dims)[0], err_msg=f"field {i}")
