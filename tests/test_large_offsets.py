"""Offsets in fields of more than 2^31 cells or rows, by the host build of the
code the kernels and launchers use (no such field is allocated)."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    out = tmp_path_factory.mktemp("index") / "libindex_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "distance-occlusion_b200", "csrc"),
                    os.path.join(ROOT, "tests", "index_host.cpp"), "-o", str(out)], check=True)
    L = C.CDLL(str(out))
    L.host_edt_x_bytes.restype = L.host_edt_bytes.restype = C.c_size_t
    return L


@pytest.mark.parametrize("w,h,d", [(1024, 2048, 1025), (37, 70000, 3000), (1, 50000, 50000), (8, 4, 3)])
def test_cells_of_a_mask_word(host, w, h, d):
    ws = (w + 31) // 32
    words = ws * h * d
    for wid in (0, 1, ws, words // 2, words - ws, words - 1):
        first, n = C.c_longlong(), C.c_int()
        host.host_word_cells(C.c_longlong(wid), w, C.byref(first), C.byref(n))
        row, k = divmod(wid, ws)
        assert (first.value, n.value) == (row * w + 32 * k, min(32, w - 32 * k))
    assert first.value + n.value == w * h * d


@pytest.mark.parametrize("w,h,d", [(1, 46341, 46341), (3, 60000, 60000), (1024, 1024, 1024), (7, 5, 3)])
def test_fields_of_the_mask_edt(host, w, h, d):
    up = lambda b: (b + 255) // 256 * 256
    for pitch in (w, (w + 7) // 8 * 8):
        x = up(2 * pitch * h * d)
        assert host.host_edt_x_bytes(pitch, h, d) == x
        assert host.host_edt_bytes(3, pitch, h, d) == x + 4 * pitch * h * d
        assert host.host_edt_bytes(2, pitch, h, d) == up(2 * pitch * h)
