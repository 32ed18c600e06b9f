"""Batch items at the widths where the kernel changes its engine (cells per lane,
a warp or a group of warps per row, slices in shared memory or not) equal the
per-item calls, which equal the oracle."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

IMAGES = [(1, 1), (5, 1), (64, 40), (65, 31), (128, 70), (129, 33), (256, 20), (257, 45), (512, 33), (513, 40), (1024, 37)]
VOLUMES = [(1, 1, 2), (3, 1, 9), (33, 15, 7), (64, 64, 6), (65, 17, 9), (128, 128, 5), (127, 33, 4), (129, 20, 5),
           (100, 250, 3), (300, 18, 4), (600, 9, 3)]


class Item(C.Structure):
    _fields_ = [("w", C.c_int), ("h", C.c_int), ("d", C.c_int), ("reserved", C.c_int),
                ("mask_word_offset", C.c_longlong), ("delta_byte_offset", C.c_longlong), ("dist_offset", C.c_longlong)]


@pytest.mark.parametrize("warps", [16, 8])
def test_engine_edges(dol, O, cuda, warps):
    torch = cuda
    L = dol.lib()
    rng = np.random.default_rng(3)
    dims = [d + (1,) for d in IMAGES] + VOLUMES
    items = (Item * len(dims))()
    masks, words, dbytes, cells = [], 0, 0, 0
    for i, (w, h, d) in enumerate(dims):
        shape = (h, w) if d == 1 else (d, h, w)
        b = rng.random(shape) < (0.02 if i % 2 else 0.4)
        masks.append(O.bool_to_mask(b))
        items[i] = Item(w, h, d, 0, words, dbytes, cells)
        words += len(masks[-1])
        dbytes += (w * h * d * (4 if d == 1 else 6) + 15) // 16 * 16
        cells += w * h * d
    md = torch.from_numpy(np.concatenate(masks).view(np.int32)).cuda()
    deltas = torch.zeros(dbytes, dtype=torch.uint8, device="cuda")
    dist = torch.zeros(cells, dtype=torch.float32, device="cuda")
    L.dol_tune_set(6, 1024, 8 if warps == 8 else 0)
    try:
        dol.check(L.dol_batch_sdf(len(dims), items, C.c_void_p(md.data_ptr()), C.c_void_p(deltas.data_ptr()),
                                  C.c_void_p(dist.data_ptr()), None, C.c_size_t(0), None))
        dol.sync()
        torch.cuda.synchronize()
    finally:
        L.dol_tune_set(6, 1024, 0)
    got_d, got_f = deltas.cpu().numpy(), dist.cpu().numpy()
    for i, (w, h, d) in enumerate(dims):
        dm = (w, h) if d == 1 else (w, h, d)
        want = O.propagate("danielsson", O.border_init(masks[i], dm), dm, 2)
        n = w * h * d
        g = got_d[items[i].delta_byte_offset:][:n * (4 if d == 1 else 6)].view(np.int16).reshape(want.shape)
        np.testing.assert_array_equal(g, want, err_msg=f"{dm}")
        f = O.deltas_to_dist(want, dm, 2, masks[i])
        assert np.array_equal(got_f[items[i].dist_offset:][:n].view(np.uint32), f.reshape(-1).view(np.uint32)), dm
