"""Forward steps by marches along x (SWD_OPT_MARCH) against the two step kernels: the same bits.

The march runs on grids that fill the L2 only, so the grids are large and the records short.  Rows:
the last row tile full and with one row left; columns: chunks that end inside and outside the
frame; two edge wells and receivers scattered over the padded grid (frame cells, duplicates); the
source inside the strip band and in the frame corner; odd and even step counts (the fields are
double-buffered), fewer and more steps than a captured chunk; FP32 and 16-bit strips."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    # nx, nz, pml, nt, strips
    "f32_odd": (3001, 1509, 13, 67, "STRIP_F32"),        # 1543 rows = 13 full tiles of 112 and 87
    "f16_even": (3333, 1422, 13, 130, "STRIP_F16"),      # 1456 rows: exactly 13 tiles
    "i16_short": (3100, 1423, 13, 45, "STRIP_I16"),      # one row in the last tile
    "tall": (1201, 4003, 30, 65, "STRIP_F32"),           # few lean chunks along x
}


@pytest.mark.parametrize("name", list(CASES))
def test_march_same_bits(swd, name):
    nx, nz, pml, nt, prec = CASES[name]
    rng = np.random.default_rng(9)
    pmlc = pml + 4
    v = (1900.0 + 900.0 * np.arange(nz)[None, :] / nz + rng.uniform(-80, 80, (nx, 1))).astype(np.float32)
    vp = swd.pad_model(v, pmlc)
    ntx, ntz = vp.shape
    E = swd.Engine(nx, nz, pml, 4, 5.0, 5.0, 5e-4, nt)
    E.setup_default(vp, (1000.0 + rng.uniform(-50, 50, vp.shape)).astype(np.float32))
    E.set_strip_precision(getattr(swd, prec))
    n = 80
    rix, riz = rng.integers(0, ntx, n).astype(np.int32), rng.integers(0, ntz, n).astype(np.int32)
    rix[:40] = pmlc + nx // 2
    riz[:40] = pmlc + np.arange(40)
    riz[1] = riz[0]
    rick = swd.ricker_wave(nt, 40.0, 5e-4)
    data = rng.standard_normal((n, nt)).astype(np.float32)
    out = {}
    for march in (0, 1):
        E.set_option(swd.OPT_MARCH, march)
        n0, r = E.launch_count(), []
        for sx, sz in ((pmlc + nx // 2, pmlc + 1), (3, ntz - 5)):
            s = swd.ShotSpec(sx, sz, rix, riz, nt)
            r.append(E.rtm_forward(s, rick, syn=True))
            E.rtm_backward(s, data, flags=swd.RTM_PREPROCESS | swd.RTM_NO_STACK, want=())
            r += list(E.rtm_raw()[:2])   # the reconstruction starts from the march's state and strips
            r.append(E.forward(s, rick))
        out[march] = (r, E.launch_count() - n0)
    assert out[1][1] < out[0][1] - 3 * nt               # one launch per forward step instead of two
    for i, (a, b) in enumerate(zip(out[1][0], out[0][0])):
        assert i >= len(out[0][0]) // 2 or np.abs(b).max() > 0, i
        assert np.array_equal(a, b), i


def test_march_needs_a_large_grid(swd):
    """Grids that stay in L2, other stencil lengths and host-launched steps keep the two kernels."""
    for nx, nz, Lc, graphs in ((1201, 601, 4, 1), (3001, 1509, 5, 1), (3001, 1509, 4, 0)):
        nt = 66
        E = swd.Engine(nx, nz, 10, Lc, 5.0, 5.0, 5e-4, nt)
        E.set_option(swd.OPT_GRAPHS, graphs)
        vp = np.full((nx + 2 * (10 + Lc), nz + 2 * (10 + Lc)), 2000.0, np.float32)
        E.setup_default(vp, np.full_like(vp, 1000.0))
        s = swd.ShotSpec(60, 60, np.array([70], np.int32), np.array([60], np.int32), nt)
        n0 = E.launch_count()
        E.rtm_forward(s, swd.ricker_wave(nt, 25.0, 5e-4))
        assert E.launch_count() - n0 >= 2 * nt


def test_flat_grid_keeps_the_step_kernels(swd):
    """A large grid that is nearly all frame: the march would take 1.6 times as long."""
    nx, nz, pml, nt = 36000, 100, 10, 64
    E = swd.Engine(nx, nz, pml, 4, 5.0, 5.0, 5e-4, nt)
    vp = np.full((nx + 28, nz + 28), 2000.0, np.float32)
    E.setup_default(vp, np.full_like(vp, 1000.0))
    s = swd.ShotSpec(60, 60, np.array([70], np.int32), np.array([60], np.int32), nt)
    n0 = E.launch_count()
    E.forward(s, swd.ricker_wave(nt, 25.0, 5e-4))
    assert E.launch_count() - n0 >= 2 * nt
