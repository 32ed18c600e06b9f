"""Batch items at the lines where an item's rows change hands: images of less than
64 cells (rows in registers or in shared memory, several rows of distances at a
time), volumes whose slices do not fit in shared memory, volumes of wide rows by
a CTA.  Against the oracle."""
import numpy as np
import pytest

from test_gpu_batch_shapes import Item

pytestmark = pytest.mark.gpu

DIMS = [(1, 50, 1), (2, 77, 1), (15, 40, 1), (16, 41, 1), (17, 40, 1), (31, 30, 1), (32, 31, 1), (33, 30, 1), (63, 31, 1),
        (64, 30, 1), (100, 45, 1), (127, 30, 1), (129, 30, 1), (20, 600, 3), (32, 560, 2), (33, 560, 3), (64, 560, 2),
        (65, 300, 3), (127, 300, 2), (128, 300, 2), (200, 20, 3), (257, 6, 4), (512, 5, 3), (513, 4, 4), (1024, 3, 3)]


@pytest.mark.parametrize("warps", [16, 8])
@pytest.mark.parametrize("copies", [1, 120])   # few items per CTA; more than a CTA takes one at a time
def test_items(dol, O, cuda, warps, copies):
    import ctypes as C
    torch = cuda
    rng = np.random.default_rng(warps)
    kinds = []
    for i, (w, h, d) in enumerate(DIMS):
        dm = (w, h) if d == 1 else (w, h, d)
        m = O.bool_to_mask(rng.random(tuple(reversed(dm))) < (0.02 if i % 2 else 0.4))
        want = O.propagate("danielsson", O.border_init(m, dm), dm, 2)
        kinds.append((m, want.reshape(-1), O.deltas_to_dist(want, dm, 2, m).reshape(-1).view(np.uint32)))
    n = len(DIMS) * copies
    items = (Item * n)()
    words = dbytes = cells = 0
    for i in range(n):
        w, h, d = DIMS[i % len(DIMS)]
        items[i] = Item(w, h, d, 0, words, dbytes, cells)
        words += len(kinds[i % len(DIMS)][0])
        dbytes += (w * h * d * (4 if d == 1 else 6) + 3) // 4 * 4
        cells += w * h * d
    md = torch.from_numpy(np.concatenate([k[0] for k in kinds] * copies).view(np.int32)).cuda()
    deltas = torch.zeros(dbytes, dtype=torch.uint8, device="cuda")
    dist = torch.zeros(cells, dtype=torch.float32, device="cuda")
    L = dol.lib()
    L.dol_tune_set(6, 1024, 8 if warps == 8 else 0)
    try:
        dol.check(L.dol_batch_sdf(n, items, C.c_void_p(md.data_ptr()), C.c_void_p(deltas.data_ptr()),
                                  C.c_void_p(dist.data_ptr()), None, C.c_size_t(0), None))
        dol.sync()
    finally:
        L.dol_tune_set(6, 1024, 0)
    got_d, got_f = deltas.cpu().numpy(), dist.cpu().numpy().view(np.uint32)
    for i in range(n):
        _, d, f = kinds[i % len(DIMS)]
        assert np.array_equal(got_d[items[i].delta_byte_offset:][:2 * len(d)].view(np.int16), d), DIMS[i % len(DIMS)]
        assert np.array_equal(got_f[items[i].dist_offset:][:len(f)], f), DIMS[i % len(DIMS)]
