"""Model smoothing with every kind of window against its definition in double precision on the host:
the same sums in the same order, so the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _smooth(v, pml, w):
    """Gaussian of 2 w + 1 taps per axis, double sums row by row of the window, indices clamped; the first
    eight rows under the frame unchanged; the frame filled from the edges, x first."""
    ntx, ntz = v.shape
    k = np.arange(-w, w + 1)
    s = w / 2.0
    c = 1.0 / (2.0 * 3.1415926 * s * s) * np.exp(-(k[:, None] ** 2 + k[None, :] ** 2) / (2.0 * s * s))
    total = 0.0
    for t in c.ravel():
        total += t
    c = c / total
    x, z = np.arange(pml, ntx - pml), np.arange(pml, ntz - pml)
    acc = np.zeros((len(x), len(z)))
    d = v.astype(np.float64)
    for a in range(2 * w + 1):                # rows
        zz = np.clip(z - w + a, 0, ntz - 1)
        for b in range(2 * w + 1):            # columns
            acc = acc + d[np.clip(x - w + b, 0, ntx - 1)][:, zz] * c[a, b]
    out = v.copy()
    out[np.ix_(x, z[z >= pml + 8])] = acc.astype(np.float32)[:, z >= pml + 8]
    out[:pml, pml:ntz - pml] = out[pml, pml:ntz - pml]
    out[ntx - pml:, pml:ntz - pml] = out[ntx - pml - 1, pml:ntz - pml]
    out[:, :pml] = out[:, pml:pml + 1]
    out[:, ntz - pml:] = out[:, ntz - pml - 1:ntz - pml]
    return out


@pytest.mark.parametrize("window", [1, 5, 24, 25, 33, 64])
def test_windows(swd, window):
    """Either side of the widths where the kernel stops to use a tile in shared memory, on a grid with
    ragged blocks.  (The weights' exp may differ from numpy's in the last place: 1e-6 of the value.)"""
    rng = np.random.default_rng(window)
    v = (2000.0 + 500.0 * rng.random((107, 121))).astype(np.float32)
    E = swd.Engine(64, 64, 8, 4, 5.0, 5.0, 5e-4, 64)
    got, ref = E.smooth(v, 9, window), _smooth(v, 9, window)
    assert np.max(np.abs(got / ref - 1.0)) < 1e-6
    assert np.array_equal(got[:, :17], ref[:, :17])   # rows that are only copied


def test_tile_and_memory_taps_same_bits(swd):
    """A window that takes the tile on large grids only: the interior of a large grid against the same
    cells of a small one cut out of it."""
    w, pml = 28, 10
    rng = np.random.default_rng(0)
    v = (2000.0 + 500.0 * rng.random((1420, 760))).astype(np.float32)
    E = swd.Engine(64, 64, 8, 4, 5.0, 5.0, 5e-4, 64)
    big, small = E.smooth(v, pml, w), E.smooth(v[200:420, 100:400], pml, w)
    cut = (slice(w + pml, 220 - w - pml), slice(w + pml, 300 - w - pml))
    assert np.array_equal(big[200:420, 100:400][cut], small[cut])
