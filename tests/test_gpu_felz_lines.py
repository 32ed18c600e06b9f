"""DOL::Felzenszwalb on float fields: the shared-memory line kernel and the
long-line form give the oracle's floats bit for bit at the edges of their
ranges (one line, one cell, lines that do not fill a CTA or a staging row, the
last length that fits in shared memory and the first that does not)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1), (1, 40), (40, 1), (7, 300), (8, 33), (149, 31), (1025, 9), (2100, 50),
                                  (3, 11400), (2, 11500), (17000, 3)])
@pytest.mark.parametrize("kind", ["heights", "spikes", "mask"])
def test_lines_match_oracle(dol, O, cuda, dims, kind):
    rng = np.random.default_rng(sum(dims))
    shape = (dims[1], dims[0])
    if kind == "heights":      # smooth plus rough: short envelopes with many pops
        f = (200 * np.sin(np.arange(dims[0]) / 17.0)[None, :] * np.cos(np.arange(dims[1]) / 23.0)[:, None]
             + 30 * rng.random(shape))
    elif kind == "spikes":     # every parabola stays, or one pops them all
        f = np.where(rng.random(shape) < 0.02, -1e6, rng.random(shape))
    else:
        f = np.where(rng.random(shape) < 0.01, 0.0, np.finfo(np.float32).max)
    f = f.astype(np.float32)
    want = O.felzenszwalb(f, dims)
    got = dol.felzenszwalb(cuda.from_numpy(f.copy()).cuda(), dims).cpu().numpy()
    assert np.array_equal(got.view(np.uint32), np.asarray(want, np.float32).view(np.uint32))


@pytest.mark.parametrize("dims", [(5, 33), (64, 97), (3, 1500), (33, 260)])
@pytest.mark.parametrize("kind", ["line", "integers", "near", "bend", "few"])
def test_lines_with_ties_match_oracle(dol, O, cuda, dims, kind):
    """Fields whose envelopes tie or nearly tie: collinear heights, small
    integers, rounding noise on a line, long slightly bent runs, whole lines
    without a site."""
    rng = np.random.default_rng(dims[0] * 7 + dims[1])
    shape = (dims[1], dims[0])
    y, x = np.mgrid[:shape[0], :shape[1]].astype(np.float64)
    if kind == "line":         # heights along both passes on one line: everything pops
        f = 3 * y - y * y
    elif kind == "integers":
        f = rng.integers(0, 60, shape) * 1.0
    elif kind == "near":       # the line plus noise of a unit in the last place
        f = 0.1 * y + 1000.3 - y * y
    elif kind == "bend":       # convex by a little, in runs
        f = 1e-4 * (y % 40) ** 2 - y * y
    else:
        f = np.where((rng.random(shape) < 0.02) & (x % 5 < 2), rng.random(shape), np.finfo(np.float32).max)
    f = f.astype(np.float32)
    want = O.felzenszwalb(f, dims)
    got = dol.felzenszwalb(cuda.from_numpy(f.copy()).cuda(), dims).cpu().numpy()
    assert np.array_equal(got.view(np.uint32), np.asarray(want, np.float32).view(np.uint32))
