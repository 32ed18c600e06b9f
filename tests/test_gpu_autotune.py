"""dol_autotune ends at the built-in rule unless something else is faster: every
family's untuned launch is one of its candidates, also after another value was
kept, and what it keeps is no slower than no tuning."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DAN2, DAN3, FS2, FS3, JFA2, JFA3, BATCH, EDT, ROWS, SLICES = range(10)


@pytest.fixture
def tuned(dol):
    L = dol.lib()
    touched = []

    def run(kind, dims, before=0):
        w, h, d = dims if len(dims) == 3 else dims + (1,)
        touched.append((kind, w))
        L.dol_tune_set(kind, w, before)
        dol.check(L.dol_autotune(kind, w, h, d, None))
        return L.dol_tune_get(kind, w)
    yield run
    for kind, w in touched:
        L.dol_tune_set(kind, w, 0)


def test_jumpflood_2d_can_stay_one_launch(tuned):
    assert tuned(JFA2, (512, 512)) == 0
    assert tuned(JFA2, (512, 512), before=16) == 0


def test_fastsweep_3d_returns_to_the_columns(tuned):
    assert tuned(FS3, (128, 128, 128), before=-2) > 0   # (the wavefront takes several times as long)
    assert tuned(FS3, (1024, 3, 3), before=1) <= 0      # the slices of the rule, or the wavefront: not the columns


@pytest.mark.parametrize("kind,dims", [(ROWS, (200, 160, 30)), (ROWS, (300, 200)), (SLICES, (200, 160, 30))])
def test_danielsson_blocks(tuned, kind, dims):
    allowed = {ROWS: {0, 4, 8, 16, 65536}, SLICES: {0, 1, 4, 16, 64}}[kind]
    assert tuned(kind, dims, before=16) in allowed


@pytest.mark.parametrize("kind,method,dims", [(DAN3, "danielsson", (256, 256, 64)), (DAN2, "danielsson", (1024, 1024)),
                                              (FS2, "fastsweep", (600, 200)), (JFA3, "jumpflood", (128, 128, 128))])
def test_tuned_is_no_slower(dol, O, cuda, tuned, kind, method, dims):
    torch = cuda
    L = dol.lib()
    rng = np.random.default_rng(5)
    b = np.zeros(dims[::-1], bool)
    for _ in range(30):   # boxes
        at = [rng.integers(0, s) for s in b.shape]
        b[tuple(slice(a, a + int(rng.integers(3, 30))) for a in at)] = True
    md = torch.from_numpy(O.bool_to_mask(b).view(np.int32)).cuda()
    start = dol.init_border(md, dims)

    def best():
        t = []
        for _ in range(5):
            work = start.clone()
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            dol.propagate(method, work, dims, 2)
            e[1].record()
            e[1].synchronize()
            t.append(e[0].elapsed_time(e[1]))
        return min(t), work

    untuned, want = best()
    value = tuned(kind, dims)
    L.dol_tune_set(kind, dims[0], value)
    now, got = best()
    assert torch.equal(got, want)
    assert now <= 1.15 * untuned, value   # (another content than the tuner's: 15 % covers what that changes)
