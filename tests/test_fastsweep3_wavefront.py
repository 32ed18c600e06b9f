"""FastSweep 3D's anti-diagonal wavefront: the table of its diagonals, and calls of
different shapes queued one behind the other, each with its own table."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_rows_before_a_diagonal(tmp_path):
    out = tmp_path / "libdiagonals.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "distance-occlusion_b200", "csrc"),
                    os.path.join(ROOT, "tests", "diagonals_host.cpp"), "-o", str(out)], check=True)
    f = C.CDLL(str(out)).host_rows_before_diagonal
    for H, D in ((1, 1), (1, 7), (9, 1), (4, 4), (5, 12), (13, 6), (300, 41)):
        jj, kk = np.mgrid[1:H + 1, 1:D + 1]
        s = (jj + kk).ravel()
        assert [f(H, D, c) for c in range(H + D + 2)] == [int((s < c).sum()) for c in range(H + D + 2)]
    assert f(40000, 50000, 90001) == 40000 * 50000


@pytest.mark.gpu
def test_calls_queued_one_behind_the_other(dol, O, cuda):
    torch = cuda
    L = dol.lib()
    rng = np.random.default_rng(2)
    shapes = [(40, 60, 50), (33, 5, 9), (40, 9, 70), (50, 30, 4), (64, 3, 3), (35, 80, 20)]
    L.dol_tune_set(3, 64, -2)   # the bucket of widths 33 .. 64
    try:
        fields, got = [], []
        for dims in shapes:
            m = O.bool_to_mask(rng.random(dims[::-1]) < 0.05)
            fields.append(O.border_init(m, dims))
        on_gpu = [torch.from_numpy(f.copy()).cuda() for f in fields]
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)   # the stream is busy while all of them are queued
        for dims, t in zip(shapes, on_gpu):
            dol.fastsweep(t, dims, 2)
        dol.sync()
        for dims, f, t in zip(shapes, fields, on_gpu):
            np.testing.assert_array_equal(t.cpu().numpy(), O.propagate("fastsweep", f, dims, 2), err_msg=f"{dims}")
    finally:
        L.dol_tune_set(3, 64, 0)
