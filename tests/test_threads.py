"""Engines of several threads at the same time: what one thread's call sets up for its launches must
not be changed under them by another's."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_smoothing_windows_of_two_threads(swd):
    """Small and large windows (different amounts of shared memory) side by side."""
    rng = np.random.default_rng(1)
    v = (2000.0 + 500.0 * rng.random((120, 100))).astype(np.float32)
    windows = (2, 40, 5, 24)
    made = [swd.Engine(64, 64, 8, 4, 5.0, 5.0, 5e-4, 64) for _ in windows]
    ref = [E.smooth(v, 14, w) for E, w in zip(made, windows)]

    def many(k):
        return all(np.array_equal(made[k].smooth(v, 14, windows[k]), ref[k]) for _ in range(300))

    with ThreadPoolExecutor(len(windows)) as pool:
        assert all(pool.map(many, range(len(windows))))


def test_deconvolution_geometries_of_two_threads(swd):
    """Windows of very different widths side by side."""
    rng = np.random.default_rng(2)
    geo = [((11, 11), (21, 21), (5, 5)), ((21, 21), (101, 101), (20, 20)), ((15, 15), (61, 61), (12, 12))]
    mig = rng.standard_normal((180, 170)).astype(np.float32)
    made = [swd.Engine(64, 64, 8, 4, 5.0, 5.0, 5e-4, 64) for _ in geo]
    psf = []
    for (w, _), _, _ in geo:
        p = np.zeros(mig.shape, np.float32)
        p[w // 2::w, w // 2::w] = 1.0
        p[w // 2 + 1::w, w // 2::w] = 0.3
        psf.append(p)

    def one(k):
        return made[k].decon(mig, psf[k], *geo[k], 1e-3)[0]

    ref = [one(k) for k in range(len(geo))]

    def many(k):
        return all(np.array_equal(one(k), ref[k]) for _ in range(150))

    with ThreadPoolExecutor(len(geo)) as pool:
        assert all(pool.map(many, range(len(geo))))
