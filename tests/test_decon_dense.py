"""The deconvolution's windows as real matrix products (decon_dense.cuh) against the FP64 oracle and
against the chirp-z FFT windows, which swd_decon_noalloc still runs.

Geometries at the edges of the plan: the smallest windows, axes with different patch sizes but one
transform length, even transform lengths that differ per axis (a frequency that is its own
negative), PSFs blended per window, one PSF per window because the lattice has more points than
there are windows, output windows that need two tiles per thread, the widest windows that fit in
shared memory and windows that do not (FFT path).

Tolerance: both paths form sums of at most 250 single-precision products per axis and divide by a
denominator damped to 1e-3 of the peak power, so single-precision roundings (6e-8 each, random)
come out at a few 1e-6; 2e-5 leaves room for the damping, 1e-4 of any structural error is seen."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 2e-5
CASES = {
    # nx, nz, psf, filter, snap, fft_n, psf_interp
    "smallest": (60, 70, (3, 3), (5, 5), (2, 2), (0, 0), 0),
    "odd_axes": (150, 171, (11, 15), (29, 25), (5, 4), (0, 0), 0),
    "even_lengths": (140, 133, (11, 9), (31, 27), (5, 4), (64, 40), 0),
    "one_even": (140, 133, (11, 9), (31, 27), (5, 4), (45, 40), 1),
    "blended": (230, 200, (21, 21), (41, 41), (9, 9), (0, 0), 1),
    "psf_per_window": (120, 130, (7, 7), (61, 61), (28, 28), (0, 0), 0),
    "two_tiles": (400, 380, (31, 31), (141, 141), (67, 67), (0, 0), 0),
    "widest": (750, 720, (99, 99), (139, 139), (54, 54), (0, 0), 0),
    "too_wide": (420, 400, (41, 41), (201, 201), (60, 60), (0, 0), 0),
}


def _inputs(nx, nz, psf, seed):
    rng = np.random.default_rng(seed)
    mig = rng.standard_normal((nx, nz)).astype(np.float32)
    img = np.zeros((nx, nz), np.float32)
    img[psf[0] // 2::psf[0], psf[1] // 2::psf[1]] = 1.0
    img[psf[0] // 2 + 1::psf[0], psf[1] // 2::psf[1]] = rng.uniform(-0.5, 0.5, img[psf[0] // 2 + 1::psf[0], psf[1] // 2::psf[1]].shape)
    return mig, img


@pytest.mark.parametrize("name", list(CASES))
def test_dense_windows_match_oracle(swd, orc, name):
    nx, nz, psf, flt, snap, fft_n, interp = CASES[name]
    mig, img = _inputs(nx, nz, psf, 31)
    dec, coef = swd.decon(mig, img, psf, flt, snap, 1e-3, fft_n=fft_n, psf_interp=interp)
    odec, ocoef = orc.decon(nx, nz, mig, img, psf, flt, snap, 1e-3, fft_n=fft_n, psf_interp=interp)
    assert np.array_equal(coef, ocoef)
    assert rel_l2(dec, odec) < TOL


def test_dense_windows_match_fft_windows_and_zero_psf(swd):
    """Against the FFT windows on the same arrays, one lattice PSF being all zero: its windows come
    out as NaN (0/0 in the normalisation) on both paths, all others agree."""
    import torch
    nx, nz, psf, flt, snap = 300, 290, (11, 11), (31, 31), (7, 7)
    mig, img = _inputs(nx, nz, psf, 32)
    img[15 * 11:16 * 11, 12 * 11:13 * 11] = 0.0
    p = swd.DeconParams(nx, nz, *psf[:1], psf[1], flt[0], flt[1], snap[0], snap[1], 1e-3, 0, 0)
    d = [torch.from_numpy(a).cuda() for a in (mig, img)]
    out = [torch.zeros((nx, nz), device="cuda") for _ in range(2)]
    L = swd.lib()
    L.swd_decon_noalloc.argtypes = [C.POINTER(swd.DeconParams)] + [C.c_void_p] * 5
    assert L.swd_decon_noalloc(C.byref(p), d[0].data_ptr(), d[1].data_ptr(), out[0].data_ptr(), out[1].data_ptr(),
                               torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    ref = out[0].cpu().numpy()
    dec, _ = swd.decon(mig, img, psf, flt, snap, 1e-3)
    assert np.isnan(ref).any() and np.array_equal(np.isnan(dec), np.isnan(ref))
    ok = ~np.isnan(ref)
    assert rel_l2(dec[ok], ref[ok]) < TOL
