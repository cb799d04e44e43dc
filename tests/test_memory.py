"""Calls on a device whose memory is nearly full: scratch that only makes a call faster must not make
it, or a later one, fail."""
import ctypes as C

import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu

MB = 1 << 20


class Filled:
    """The device's memory taken but for `leave` bytes."""

    def __init__(self, leave):
        self.leave = int(leave)

    def __enter__(self):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        n = torch.cuda.mem_get_info()[0] - self.leave
        assert n > 0
        self.t = torch.empty(n // (2 * MB) * 2 * MB, dtype=torch.uint8, device="cuda")

    def __exit__(self, *exc):
        del self.t
        torch.cuda.empty_cache()


class Decon:
    """A device-resident deconvolution whose matrix-product windows want 148 MB of scratch (a PSF blend per
    window) beside the 19 MB that every path needs."""

    def __init__(self, swd):
        nx, nz, w, f, s = 1601, 801, 79, 79, 24
        rng = np.random.default_rng(5)
        img = torch.zeros(nx, nz, device="cuda")
        img[w // 2::w, w // 2::w] = 1.0
        img[w // 2 + 1::w, w // 2::w] = 0.4
        self.ins = (torch.from_numpy(rng.standard_normal((nx, nz)).astype(np.float32)).cuda(), img)
        self.out = (torch.zeros_like(img), torch.zeros_like(img))
        self.prm = swd.DeconParams(nx, nz, w, w, f, f, s, s, 1e-3, 0, 0, 1)
        self.swd = swd

    def __call__(self, E):
        E._ck(self.swd.lib().swd_decon(E._h, C.byref(self.prm), *[self.swd._ptr(t) for t in self.ins + self.out]))
        return self.out[0].cpu().numpy()


def test_decon_falls_back_to_the_fft_windows(swd):
    job = Decon(swd)
    E = swd.Engine(64, 64, 8, 4, 5.0, 5.0, 5e-4, 64)
    job.prm.iters = 1                                   # the FFT kernels are loaded
    job(E)
    job.prm.iters = 0
    ref = job(E)
    E.close()
    E = swd.Engine(64, 64, 8, 4, 5.0, 5.0, 5e-4, 64)
    with Filled(152 * MB):
        got = job(E)
    assert not np.array_equal(got, ref)                 # the other path
    assert rel_l2(got, ref) < 2e-5                      # (single-precision roundings of both, as between them elsewhere)
    assert np.array_equal(job(E), ref)                  # and back, with the memory back
