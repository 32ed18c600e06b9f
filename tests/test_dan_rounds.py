"""The Danielsson block iteration on deltas a caller brings, not only those a
mask gives: random components of several sizes and densities on small fields
of several x blocks.  On the CPU a serial model of the iteration equals the
oracle's sweeps and stays within the kernel's limit of rounds (csrc/dan_rounds.h);
on the GPU the entries give the oracle's deltas."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHAPES = [(65, 8, 2), (130, 4, 3), (100, 4, 3), (65, 3, 6), (500, 4, 3), (70, 30, 1), (300, 5, 1)]


def fields(dims, seed, count):
    """int16 deltas: components up to `size`, cells at max elsewhere"""
    w, h, d = dims
    n = 2 if d == 1 else 3
    far = 8192 if d == 1 else 25000
    rng = np.random.default_rng(seed)
    for i in range(count):
        size = (6, 100, 100, 2000)[i % 4]
        f = rng.integers(-size, size + 1, (d, h, w, n)).astype(np.int16)
        f[rng.random((d, h, w)) >= (0.05, 0.3, 1.0)[i % 3]] = far
        yield np.ascontiguousarray(f if d > 1 else f[0])


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    out = tmp_path_factory.mktemp("danrounds") / "libdan_rounds.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "distance-occlusion_b200", "csrc"),
                    os.path.join(ROOT, "tests", "dan_rounds_host.cpp"), "-o", str(out)], check=True)
    return C.CDLL(str(out))


def test_rounds_stay_within_the_limit(O, model):
    over_block_count = 0
    for s, dims in enumerate(SHAPES):
        w, h, d = dims
        odims = dims if d > 1 else dims[:2]
        for i, f in enumerate(fields(dims, s, 60)):
            cw = 1 + i % 2
            want = O.propagate("danielsson", f, odims, cw)
            got = f.copy()
            left, blocks = C.c_longlong(), C.c_int()
            rounds = model.dan_rounds_model(3 if d > 1 else 2, w, h, d, cw, 4 if d > 1 else 8, 2, 64,
                                            got.ctypes.data_as(C.c_void_p), C.byref(left), C.byref(blocks))
            np.testing.assert_array_equal(got, want, err_msg=f"{dims} field {i}")
            assert left.value >= 0, f"{dims} field {i}: {rounds} rounds"
            over_block_count += rounds > 4 * blocks.value + 8
    assert over_block_count > 0   # a limit by the number of blocks would have cut some of these short


def test_limit_of_large_fields(model):
    """64-bit arithmetic, and below 2^28 (the state word's room for a round)"""
    f = model.dan_rounds_limit
    f.argtypes = [C.c_longlong] * 3
    assert f(1, 8, 3) == 98
    for args in ((1 << 20, 1 << 20, 1), (2**31 - 1, 2**31 - 1, 64), (65535, 16384, 32), (1, 2**31 - 1, 1)):
        assert 1 << 27 < f(*args) < 1 << 28


@pytest.fixture
def tune_rows(dol):
    set_ = []

    def put(w, rows):
        set_.append(w)
        dol.lib().dol_tune_set(8, w, rows)   # DOL_TUNE_DANIELSSON_ROWS
    yield put
    for w in set_:
        dol.lib().dol_tune_set(8, w, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [0, 4])   # the engine that the shape gets; blocks of 4 rows
@pytest.mark.parametrize("dims", SHAPES)
def test_callers_deltas(dol, O, cuda, tune_rows, dims, rows):
    d = dims[2]
    tune_rows(dims[0], rows)
    odims = dims if d > 1 else dims[:2]
    for i, f in enumerate(fields(dims, 100 + sum(dims), 48)):
        cw = 1 + i % 2
        t = cuda.from_numpy(f).cuda()
        dol.danielsson(t, odims, cw)
        dol.sync()
        np.testing.assert_array_equal(t.cpu().numpy(), O.propagate("danielsson", f, odims, cw), err_msg=f"field {i}")
