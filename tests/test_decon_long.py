"""Deconvolution of an image with more rows than a grid of blocks of 256 has room for in its second
dimension (65,535 blocks)."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_image_of_seventeen_million_rows(swd):
    """An image and PSFs that repeat every lattice cell: away from its ends the long image's result is, bit
    for bit, a short one's at the same place of the cell."""
    nx, w = 21, 3
    cell = torch.tensor([[0.2, -0.1, 0.3], [1.0, 2.0, -0.7], [0.4, 0.1, 0.6]], device="cuda")
    pcell = torch.tensor([[0.1, 0.0, 0.05], [0.2, 1.0, -0.1], [0.0, 0.15, 0.0]], device="cuda")
    E = swd.Engine(64, 64, 8, 4, 5.0, 5.0, 5e-4, 64)

    def run(nz):
        mig, psf = (c.repeat(nx // w, nz // w) for c in (cell, pcell))
        prm = swd.DeconParams(nx, nz, w, w, 5, 5, 2, 2, 1e-3, 0, 0)
        dec, coef = torch.zeros_like(mig), torch.zeros_like(mig)
        E._ck(swd.lib().swd_decon(E._h, C.byref(prm), *[swd._ptr(t) for t in (mig, psf, dec, coef)]))
        return dec, coef

    long, short = run(65535 * 256 + 903), run(903)
    assert long[0].shape[1] > 65535 * 256 and short[0].abs().max() > 0
    for a, b in zip(long, short):
        assert torch.equal(a[:, 65535 * 256 - 300:65535 * 256 + 300], b[:, 150:750])
    E.close()
