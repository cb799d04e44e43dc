"""Steps that stream from HBM: operands prefetched ahead, and scattered fields that read the perturbed
model only where it differs."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

# perturbed cells of the padded 68 x 178 grid: rows at the edges of a warp's 128, columns at the edges
# of a block's 8 and of the grid, scatterers in the frame, one array only, everywhere
WHERE = {
    "row_127": (slice(30, 31), slice(127, 128), "rho"),
    "row_128": (slice(32, 33), slice(128, 129), "rho"),
    "vp_only": (slice(39, 40), slice(100, 101), "vp"),
    "lattice": (slice(16, 56, 7), slice(20, 170, 7), "rho"),
    "edge_of_grid": (slice(0, 68, 67), slice(20, 60), "rho"),
    "everywhere": (slice(0, 68), slice(0, 178), "both"),
}


@pytest.mark.parametrize("name", list(WHERE))
def test_scattered_field_vs_fp64(swd, orc, name):
    """Against the difference of two FP64 records, within the 1e-4 of the exact scattered field."""
    sx, sz, what = WHERE[name]
    nx, nz, pml, Lc, nt, h, dt = 40, 150, 10, 4, 260, 5.0, 5e-4
    p = pml + Lc
    rng = np.random.default_rng(4)
    vp = swd.pad_model((2000.0 + 5.0 * np.arange(nz)[None, :] + rng.uniform(-50, 50, (nx, nz))).astype(np.float32), p)
    rho = (1000.0 + rng.uniform(-50, 50, vp.shape)).astype(np.float32)
    vp1, rho1 = vp.copy(), rho.copy()
    if what != "vp":
        rho1[sx, sz] += 20.0
    if what != "rho":
        vp1[sx, sz] += 15.0
    ntx, ntz = vp.shape
    rix = np.concatenate([np.full(60, 25), rng.integers(4, ntx - 4, 40)]).astype(np.int32)
    riz = np.concatenate([np.arange(100, 160), rng.integers(4, ntz - 4, 40)]).astype(np.int32)
    cp, rc = orc.cpml(ntx, ntz, p, h, h, dt), orc.cal_xishu(Lc)
    rick = orc.ricker(nt, 30.0, dt)
    G = orc.Geom(30, 90, rix, riz)
    d64 = [orc.forward(orc.Model(v, r, cp, rc, p, Lc, nt, h, h, dt), G, rick, dtype=np.float64)["seis"]
           for v, r in ((vp1, rho1), (vp, rho))]
    E = swd.Engine(nx, nz, pml, Lc, h, h, dt, nt)
    E.setup_default(vp, rho)
    E.set_scatter_model(vp1, rho1)
    d = E.forward_scatter(swd.ShotSpec(30, 90, rix, riz, nt), rick)
    if not np.any(d64[0] - d64[1]):   # (the outermost columns are never updated)
        assert name == "edge_of_grid" and not np.any(d)
        return
    assert rel_l2(d, d64[0] - d64[1]) < 1e-4


@pytest.mark.parametrize("nx,nz", [(2901, 1001), (2897, 1102)])
def test_prefetched_steps_same_bits(swd, nx, nz):
    """Large grids, whose step kernels prefetch 40 columns ahead (also past the last column), against
    the kernels that do not: the backward pass in the reference's pairing, the field of a twin by the
    other kernel of a single field; the records of a perturbed model that is the model are zero."""
    nt, pml = 66, 13
    p = pml + 4
    rng = np.random.default_rng(2)
    vp = swd.pad_model((1900.0 + 900.0 * np.arange(nz)[None, :] / nz + rng.uniform(-80, 80, (nx, 1))).astype(np.float32), p)
    rho = (1000.0 + rng.uniform(-50, 50, vp.shape)).astype(np.float32)
    E = swd.Engine(nx, nz, pml, 4, 5.0, 5.0, 5e-4, nt)
    E.setup_default(vp, rho)
    ntx, ntz = vp.shape
    rix = np.full(60, ntx - 10, np.int32)
    riz = (np.arange(60) * 7 + 5).astype(np.int32)
    s = swd.ShotSpec(ntx - 30, p + 20, rix, riz, nt)
    rick = swd.ricker_wave(nt, 40.0, 5e-4)
    data = rng.standard_normal((60, nt)).astype(np.float32)
    raw = []
    for kind in (1, 0):
        E.set_option(swd.OPT_BWD_BY_KIND, kind)
        E.rtm_shot(s, rick, data, flags=swd.RTM_NO_STACK, want=())
        raw.append(list(E.rtm_raw()[:2]))
    for a, b in zip(*raw):
        assert np.abs(b).max() > 0
        assert np.array_equal(a, b)
    one = E.forward(s, rick)
    two = E.forward(s, rick, hrick=E.hilbert(rick), kz_coef=np.ones(swd.pow2(ntz), np.float32))[0]
    assert np.abs(one).max() > 0
    assert np.array_equal(one, two)
    E.set_scatter_model(vp, rho)
    assert not np.any(E.forward_scatter(s, rick))
