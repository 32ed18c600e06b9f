"""Chamfer on both sides of the number of rows from which its blocks take over, by
width, and of a block's rows, int16 and int32, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["int16", "int32"])
@pytest.mark.parametrize("w,rows", [(2, 33), (250, 33), (512, 33), (513, 24), (1024, 24), (1025, 20), (2048, 20), (2049, 16),
                                    (4096, 16)])
def test_rows(dol, O, cuda, dtype, w, rows):
    rng = np.random.default_rng(w + rows)
    top = np.iinfo(dtype).max - (4 if dtype == "int32" else 0)
    for h in (1, 2, rows - 1, rows, rows + 1, 40, 41):
        for p in (0.0, 0.003, 0.3):
            f = np.where(rng.random((h, w)) < p, rng.integers(0, 50, (h, w)), top).astype(dtype)
            t = cuda.from_numpy(f.copy()).cuda()
            assert dol.chamfer(t, (w, h)) == 3
            dol.sync()
            np.testing.assert_array_equal(t.cpu().numpy(), O.chamfer(f, (w, h))[0], err_msg=f"{h} rows")
