"""FastSweep 3D on shapes to both sides of the line between its columns and its
slices (few rows and slices of wide rows), by the rule and with the columns
chosen through the tuning table: the oracle's deltas either way, on the scratch
that the size function then gives."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(1, 2, 2), (5, 40, 3), (17, 2, 3), (17, 6, 5), (64, 9, 5), (64, 7, 9), (129, 12, 14), (129, 20, 12), (256, 12, 10),
        (257, 20, 22), (257, 22, 23), (600, 3, 4), (2048, 2, 2)]


@pytest.mark.parametrize("value", [0, 1])
@pytest.mark.parametrize("dims", DIMS)
def test_both_engines(dol, O, cuda, dims, value):
    L = dol.lib()
    rng = np.random.default_rng(sum(dims))
    fields = []
    for p in (0.003, 0.3):
        m = O.bool_to_mask(rng.random(dims[::-1]) < p)
        fields += [(O.border_init(m, dims), 2), (O.init_deltas(m, dims), 1)]
    fields.append((rng.integers(-32768, 32768, dims[::-1] + (3,)).astype(np.int16), 2))
    L.dol_tune_set(3, dims[0], value)
    try:
        ws = cuda.empty(L.dol_fastsweep_3d_workspace_size(*dims), dtype=cuda.uint8, device="cuda")
        for i, (f, cw) in enumerate(fields):
            want = O.propagate("fastsweep", f, dims, cw)
            for work in (ws, None):
                got = dol.fastsweep(cuda.from_numpy(f.copy()).cuda(), dims, cw, workspace=work)
                dol.sync()
                np.testing.assert_array_equal(got.cpu().numpy(), want, err_msg=f"field {i}")
    finally:
        L.dol_tune_set(3, dims[0], 0)


def test_few_rows_and_slices_take_the_small_scratch(dol):
    L = dol.lib()
    assert L.dol_fastsweep_3d_workspace_size(2000, 2, 2) < 4096
    assert L.dol_fastsweep_3d_workspace_size(256, 256, 256) > 256 ** 3 * 6
