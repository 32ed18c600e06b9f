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


def test_many_items(dol, O, cuda):
    """More items per CTA than it takes one at a time: wide images by groups of
    warps, then narrow ones warp by warp."""
    torch = cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(4)
    wide = [(257, 5), (300, 33), (512, 9), (513, 20), (1024, 7), (700, 2)]
    narrow = [(5, 4), (33, 6), (64, 3), (200, 5), (256, 9)]
    kinds = [(d, O.bool_to_mask(rng.random((d[1], d[0])) < p)) for d in wide + narrow for p in (0.02, 0.4)]
    which = [i % len(kinds) if i < 300 else len(kinds) - 10 + i % 10 for i in range(16 * sms + 300)]
    items = (Item * len(which))()
    masks, words, dbytes, cells = [], 0, 0, 0
    for i, k in enumerate(which):
        (w, h), m = kinds[k]
        masks.append(m)
        items[i] = Item(w, h, 1, 0, words, dbytes, cells)
        words += len(m)
        dbytes += (w * h * 4 + 15) // 16 * 16
        cells += w * h
    md = torch.from_numpy(np.concatenate(masks).view(np.int32)).cuda()
    deltas = torch.zeros(dbytes, dtype=torch.uint8, device="cuda")
    dist = torch.zeros(cells, dtype=torch.float32, device="cuda")
    dol.check(dol.lib().dol_batch_sdf(len(which), items, C.c_void_p(md.data_ptr()), C.c_void_p(deltas.data_ptr()),
                                      C.c_void_p(dist.data_ptr()), None, C.c_size_t(0), None))
    dol.sync()
    torch.cuda.synchronize()
    got_d, got_f = deltas.cpu().numpy(), dist.cpu().numpy()
    want = [(O.propagate("danielsson", O.border_init(m, d), d, 2), m, d) for d, m in kinds]
    want = [(x.reshape(-1), O.deltas_to_dist(x, d, 2, m).reshape(-1)) for x, m, d in want]
    for i, k in enumerate(which):
        d, f = want[k]
        n = items[i].w * items[i].h
        g = got_d[items[i].delta_byte_offset:][:4 * n].view(np.int16)
        assert np.array_equal(g, d.view(np.int16).reshape(-1)), (i, kinds[k][0])
        assert np.array_equal(got_f[items[i].dist_offset:][:n].view(np.uint32), f.view(np.uint32)), (i, kinds[k][0])
