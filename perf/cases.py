"""Timed workloads of the engine, through its public entry points.

Each case is one call (or one pair of calls) that a user of the framework makes: migrating a
shot, migrating a survey, modelling the data, modelling the scatter points' data, one gradient
of the least-squares migration, the windowed deconvolution of an image, the smoothing of a
velocity model.  Grids, spacings, record lengths, frames and stencil order are the ones of the
package's own configurations (configs.py) and tests; records of the larger grids are shorter
than the configurations' so that one pass stays below a second.

`prepare` makes what the caller has in hand: models, wavelets, recorded data and the engine.
`exact` repeats the arithmetic in double precision with plain torch operations and none of the
package's code, from the same single-precision inputs.
"""
from __future__ import annotations

import ctypes
import importlib
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

DEV = "cuda"


def _swd():
    """The package (its folder's name is not an identifier, so it is loaded by path)."""
    if "swd_b200" not in sys.modules:
        d = Path.cwd() / "simple-wavenumber-deconvolution_b200"
        spec = importlib.util.spec_from_file_location("swd_b200", d / "__init__.py", submodule_search_locations=[str(d)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["swd_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["swd_b200"]


# ---------------------------------------------------------------------------- the cases
def listed():
    grid = dict(pml=30, f0=25.0)
    return [
        # the smallest shot of the test suite: two edge wells, launches and latency only
        dict(name="rtm_100x60", kind="rtm", nx=100, nz=60, h=5.0, dt=5.0e-4, nt=400, pml=10, f0=25.0, wells=2, strips="f32"),
        # one shot of the small configuration
        dict(name="rtm_401x201", kind="rtm", nx=401, nz=201, h=5.0, dt=5.0e-4, nt=2000, wells=1, strips="f32", **grid),
        # one shot of the benchmark configuration's grid
        dict(name="rtm_1601x801", kind="rtm", nx=1601, nz=801, h=5.0, dt=4.0e-4, nt=2000, wells=1, strips="f32", **grid),
        # one shot of the large-survey grid with its 16-bit boundary strips
        dict(name="rtm_4001x1601", kind="rtm", nx=4001, nz=1601, h=4.0, dt=3.5e-4, nt=500, wells=1, strips="f16", **grid),
        # a walkaway survey: shots of uneven record length and aperture, batched and stacked
        dict(name="survey_1201x601", kind="survey", nx=1201, nz=601, h=5.0, dt=4.0e-4, nt=900, shots=6, **grid),
        # modelling of a shot with its Hilbert twin and the up/down separation at the well
        dict(name="model_1601x801", kind="model", nx=1601, nz=801, h=5.0, dt=4.0e-4, nt=1500, wells=1, **grid),
        # scatter-point (PSF) data of the large survey as an exact scattered field
        dict(name="scatter_4001x1601", kind="scatter", nx=4001, nz=1601, h=4.0, dt=3.5e-4, nt=450, wells=1, **grid),
        # one shot's Born data and reflectivity gradient through torch autograd
        dict(name="lsrtm_801x401", kind="lsrtm", nx=801, nz=401, h=5.0, dt=4.0e-4, nt=1000, wells=1, **grid),
        # deconvolution of an image with the reference's own window geometry, host arrays in and out
        dict(name="decon_845x702", kind="decon", nx=845, nz=702, psfwin=31, filterwin=71, snapwin=11, host=True),
        # the benchmark grid's image, arrays on the device
        dict(name="decon_1601x801", kind="decon", nx=1601, nz=801, psfwin=79, filterwin=79, snapwin=24, host=False),
        # the large survey's image, windows too large for shared memory
        dict(name="decon_4001x1601", kind="decon", nx=4001, nz=1601, psfwin=99, filterwin=129, snapwin=54, host=False),
        # the migration model: Gaussian smoothing with the reference's 11 x 11 window, host array
        dict(name="smooth_1601x801", kind="smooth", nx=1601, nz=801, pml=30, window=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rtm", "rtm", "rtm", "survey", "model", "scatter", "lsrtm", "decon", "decon", "smooth"])
    if kind == "decon":
        nx = _log(rng, 700, 4001)
        nz = max(500, min(1601, int(nx * rng.uniform(0.4, 0.9))))
        psf = rng.choice([31, 47, 63, 79, 99])
        while psf * 8 > min(nx, nz):
            psf -= 16
        flt = psf + rng.choice([0, 10, 24, 30, 40])
        flt += 1 - flt % 2
        snap = rng.randint(max(8, psf // 6), (flt - 1 - 2 * (psf // 10)) // 2)
        # the windows' step is kept at a few cells more than half of the largest listed one's
        snap = min(snap, 54)
        c = dict(kind=kind, nx=nx, nz=nz, psfwin=psf, filterwin=flt, snapwin=snap, host=rng.random() < 0.3)
        return c if _decon_windows(c) * (psf + flt) ** 2 <= 1600 * 228 ** 2 else dict(c, nx=min(nx, 901), nz=min(nz, 701))
    if kind == "smooth":
        nx = _log(rng, 100, 2000)
        return dict(kind=kind, nx=nx, nz=max(60, int(nx * rng.uniform(0.4, 0.9))), pml=rng.choice([10, 20, 30]), window=rng.randint(2, 8))
    nx = _log(rng, 100, 4001 if kind in ("rtm", "scatter") else 1601 if kind == "model" else 1001 if kind == "lsrtm" else 1201)
    nz = max(60, min(1601, int(nx * rng.uniform(0.35, 0.8))))
    pml = 10 if nx < 200 else rng.choice([20, 30])
    cells = (nx + 2 * pml + 8) * (nz + 2 * pml + 8)
    # no drawn case does more than the largest listed one: cells x steps stays below its product
    steps = {"rtm": 2.6e9, "survey": 3.0e9, "model": 2.0e9, "scatter": 3.0e9, "lsrtm": 4.0e8}[kind]
    nt = min(_log(rng, 350, 2000), max(350, int(steps / cells)))
    c = dict(kind=kind, nx=nx, nz=nz, h=rng.choice([4.0, 5.0]), dt=rng.choice([3.0e-4, 3.5e-4]), nt=nt, pml=pml, f0=rng.choice([20.0, 25.0, 30.0]))
    if kind == "survey":
        shots = rng.randint(2, 8)
        return dict(c, shots=shots, nt=max(350, min(nt, int(steps / cells / shots))))
    c["wells"] = rng.choice([1, 2])
    if kind == "rtm":
        c["strips"] = rng.choice(["f32", "f32", "i16", "f16" if nx >= 2000 else "f32"])   # 16-bit floats: large grids
    return c


# ---------------------------------------------------------------------------- inputs
LC = 4   # half stencil length of every configuration


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 12345)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _velocity(nx, nz, g):
    """Smooth random field with a depth trend and three dipping steps, 1800 to 4500 m/s."""
    low = _rand(g, 1, 1, max(4, nx // 60), max(4, nz // 60))
    f = torch.nn.functional.interpolate(low, size=(nx, nz), mode="bicubic", align_corners=True)[0, 0]
    x = torch.arange(nx, device=DEV, dtype=torch.float64)[:, None]
    z = torch.arange(nz, device=DEV, dtype=torch.float64)[None, :]
    v = 1900.0 + 900.0 * f + 900.0 * z / nz
    u = _rand(g, 3, 3).cpu().numpy()
    for k in range(3):
        v = v + (150.0 + 150.0 * u[k, 0]) * (z > (0.2 + 0.6 * u[k, 1]) * nz + (0.4 * u[k, 2] - 0.2) * (x - nx / 2))
    return v.clamp(1800.0, 4500.0)


def _box(v, n):
    h = n // 2
    a = torch.nn.functional.pad(v[None, None], (h, h, h, h), mode="replicate")
    return torch.nn.functional.avg_pool2d(a, n, stride=1)[0, 0]


def _pad(v, p):
    return torch.nn.functional.pad(v[None, None], (p, p, p, p), mode="replicate")[0, 0].float().contiguous()


def _stencil():
    """Standard staggered first-derivative weights of half length LC."""
    c = []
    for m in range(1, LC + 1):
        num = den = 1.0
        for i in range(1, LC + 1):
            if i != m:
                num *= (2 * i - 1) ** 2
                den *= (2 * m - 1) ** 2 - (2 * i - 1) ** 2
        c.append((-1) ** (m + 1) * num / abs(den) / (2 * m - 1))
    return np.array(c, np.float32)


def _cpml_axis(n, p, h, dt, half):
    """Absorbing profile of one axis: quadratic damping, frequency-shifted, frame of p cells."""
    x = (np.arange(n) + (0.5 if half else 0.0)) * h
    lo, hi, thick = p * h, (n - p - 1) * h, p * h
    d0 = -3.0 * 5500.0 * math.log(1.0e-5) / (2.0 * thick)
    depth = np.maximum(np.maximum(lo - x, x - hi), 0.0) / thick
    inside = (x > lo) & (x < hi)
    d = np.where(inside, 0.0, d0 * depth ** 2)
    al = np.where(inside, 0.0, np.maximum(math.pi * 15.0 * (1.1 - depth), 0.0))
    b = np.exp(-(d + al) * dt)
    a = np.where(d > 1.0e-6, d / np.maximum(d + al, 1.0e-30) * (b - 1.0), 0.0)
    return a.astype(np.float32), b.astype(np.float32)


def _cpml(c):
    p = c["pml"] + LC
    out = {}
    for ax, n in (("x", c["nx"] + 2 * p), ("z", c["nz"] + 2 * p)):
        for half, tag in ((False, ""), (True, "_half")):
            out[f"a_{ax}{tag}"], out[f"b_{ax}{tag}"] = _cpml_axis(n, p, c["h"], c["dt"], half)
    return out


def _ricker(nt, f0, dt):
    a = (math.pi * f0 * (np.arange(nt) * dt - 1.0 / f0)) ** 2
    return ((1.0 - 2.0 * a) * np.exp(-a)).astype(np.float32)


def _hilbert(w):
    """Hilbert transform of the wavelet on the next power of two."""
    n = 1 << (len(w) - 1).bit_length()
    f = np.fft.fft(w.astype(np.float64), n)
    s = np.where(np.arange(n) < n // 2, -1j, 1j)
    s[0] = 0.0
    return np.fft.ifft(f * s).real[:len(w)].astype(np.float32)


def _taper(c):
    nz = c["nz"] + 2 * (c["pml"] + LC)
    n = 1 << (nz - 1).bit_length()
    k = np.arange(n)
    m = int((1.0 / 15.0 / c["h"]) * (n * c["h"]))
    t = np.ones(n)
    t = np.where(k <= m, 0.5 - 0.5 * np.cos(math.pi * k / m), t)
    return np.where(k >= n - m, 0.5 + 0.5 * np.cos(math.pi * (k - n + m) / m), t).astype(np.float32)


def _reach(c, nt):
    """Cells between source and well that leave most of an nt-step record for the arrivals."""
    return max(3, min(c["nx"] // 2 - 6, int(0.25 * (nt * c["dt"] - 1.0 / c["f0"]) * 2000.0 / c["h"])))


def _wells(c, n, g=None):
    """Receiver cells (padded grid): one well in the middle over the upper 80%, or two edge wells."""
    p, nx, nz = c["pml"] + LC, c["nx"], c["nz"]
    if n == 2:
        z = np.arange(nz, dtype=np.int32) + p
        x = np.concatenate([np.full(nz, p), np.full(nz, p + nx - 1)]).astype(np.int32)
        return x, np.concatenate([z, z]).astype(np.int32)
    lo, hi = 2, int(0.8 * nz)
    if g is not None:
        r = _rand(g, 2).cpu().numpy()
        lo = 2 + int(0.05 * nz * r[0])
        hi = lo + int(nz * (0.3 + 0.3 * r[1]))
    z = np.arange(lo, hi, dtype=np.int32) + p
    return np.full(len(z), p + nx // 2, np.int32), z


def _data(c, nt, rz, f0, g):
    """Recorded traces: five events with moveout along the well and weak noise, (r_n, nt)."""
    t = torch.arange(nt, device=DEV, dtype=torch.float64)[None, :] * c["dt"]
    z = torch.as_tensor(rz, device=DEV, dtype=torch.float64)[:, None] * c["h"]
    z = z - z.min()
    T = nt * c["dt"]
    u = _rand(g, 5, 3).cpu().numpy()
    d = 0.01 * torch.randn(len(rz), nt, generator=g, device=DEV, dtype=torch.float64)
    for k in range(5):
        t0 = T * (0.1 + 0.7 * u[k, 0]) + torch.sqrt((0.3 * T * u[k, 1]) ** 2 + (z / 3000.0) ** 2) - 0.3 * T * u[k, 1]
        a = (math.pi * f0 * (t - t0)) ** 2
        d = d + (2.0 * u[k, 2] - 1.0) * (1.0 - 2.0 * a) * torch.exp(-a)
    return (1.0e-3 * d).float().contiguous()


def _grid_inputs(c, seed):
    """Everything single precision that a propagation case feeds the engine."""
    g = _gen(seed)
    p, kind = c["pml"] + LC, c["kind"]
    v = _velocity(c["nx"], c["nz"], g)
    s = dict(g=g, p=p, true=v)
    bg = _box(v, 15)
    s["vp"] = _pad(v if kind == "model" else bg, p)
    s["rho"] = (310.0 * s["vp"].double() ** 0.25).float().contiguous()
    s["rc"], s["cpml"] = _stencil(), _cpml(c)
    if kind == "survey":
        s["shots"] = []
        for k in range(c["shots"]):
            u = _rand(g, 2).cpu().numpy()
            nt = int(c["nt"] * (0.5 + 0.5 * u[0]))
            f0 = 20.0 + 15.0 * u[1]
            rx, rz = _wells(c, 1, g)
            sx = p + c["nx"] // 2 + int(_reach(c, nt) * (2.0 * (k + 0.5) / c["shots"] - 1.0))
            s["shots"].append(dict(nt=nt, sx=sx, sz=p, rx=rx, rz=rz, rick=_ricker(nt, f0, c["dt"]), data=_data(c, nt, rz, f0, g)))
        return s
    nt = c["nt"]
    s["rx"], s["rz"] = _wells(c, c["wells"])
    s["sx"] = p + (c["nx"] // 2 if c["wells"] == 1 else 0) + (-1 if c["wells"] == 1 else 1) * _reach(c, nt)
    s["sz"], s["nt"] = p, nt
    s["rick"] = _ricker(nt, c["f0"], c["dt"])
    if kind == "rtm":
        s["data"] = _data(c, nt, s["rz"], c["f0"], g)
    elif kind in ("model", "scatter"):
        s["hrick"], s["taper"] = _hilbert(s["rick"]), _taper(c)
        if kind == "scatter":   # density scatterers on a lattice: 1e-3 of vp each
            s["rho1"] = s["rho"].clone()
            at = (slice(p + 9, p + c["nx"], 19), slice(p + 5, p + c["nz"], 19))
            s["rho1"][at] += 1.0e-3 * s["vp"][at]
    elif kind == "lsrtm":
        spikes = (_rand(g, c["nx"], c["nz"]) < 0.01).double()
        s["refl"] = (0.05 * torch.randn(c["nx"], c["nz"], generator=g, device=DEV, dtype=torch.float64) * spikes).float()
        s["resid"] = _data(c, nt, s["rz"], c["f0"], g)
    return s


def _decon_geometry(c):
    full = c["filterwin"] + c["psfwin"] - 1
    out = 2 * (c["psfwin"] // 10) + 2 * c["snapwin"] + 1
    step = out - c["snapwin"]
    return full, out, step, math.ceil((c["nx"] + full) / step) + 1, math.ceil((c["nz"] + full) / step) + 1


def _decon_windows(c):
    return _decon_geometry(c)[3] * _decon_geometry(c)[4]


def _decon_inputs(c, seed):
    """Band-limited white reflectivity, and one Ricker-shaped blob of random strength per lattice point."""
    g = _gen(seed)
    mig = _box(torch.randn(c["nx"], c["nz"], generator=g, device=DEV, dtype=torch.float64), 3)
    w, h = c["psfwin"], c["psfwin"] // 2
    t = torch.arange(-7, 8, device=DEV, dtype=torch.float64) * 0.3
    r = (1 - 2 * t * t) * torch.exp(-t * t)
    cell = torch.zeros(w, w, device=DEV, dtype=torch.float64)
    cell[h - 7:h + 8, h - 7:h + 8] = r[:, None] * r[None, :]
    mx, mz = c["nx"] // w + 1, c["nz"] // w + 1
    psf = torch.kron(0.5 + _rand(g, mx, mz), cell)[:c["nx"], :c["nz"]]
    return mig.float().contiguous(), psf.float().contiguous()


EPSILON = 5.0e-4


# ---------------------------------------------------------------------------- prepare / run
STRIPS = {"f32": 0, "f16": 1, "i16": 3}


def prepare(case, seed):
    swd, kind = _swd(), case["kind"]
    if kind == "decon":
        mig, psf = _decon_inputs(case, seed)
        E = swd.Engine(64, 64, 8, LC, 5.0, 5.0, 4.0e-4, 64)
        st = dict(kind=kind, E=E, case=case, mig=mig, psf=psf)
        if case["host"]:
            st["mig"], st["psf"] = mig.cpu().numpy(), psf.cpu().numpy()
        else:
            w = (case["psfwin"], case["psfwin"], case["filterwin"], case["filterwin"], case["snapwin"], case["snapwin"])
            st["prm"] = swd.DeconParams(case["nx"], case["nz"], *w, EPSILON, 0, 0)
            st["out"] = (torch.zeros_like(mig), torch.zeros_like(mig))
        torch.cuda.synchronize()
        return st
    if kind == "smooth":
        v = _pad(_velocity(case["nx"], case["nz"], _gen(seed)), case["pml"] + LC).cpu().numpy()
        E = swd.Engine(case["nx"], case["nz"], case["pml"], LC, 5.0, 5.0, 4.0e-4, 64)
        return dict(kind=kind, E=E, vp=v, case=case)
    s = _grid_inputs(case, seed)
    torch.cuda.synchronize()
    E = swd.Engine(case["nx"], case["nz"], case["pml"], LC, case["h"], case["h"], case["dt"], case["nt"])
    E.set_stencil(s["rc"])
    E.set_cpml(s["cpml"])
    E.set_model(s["vp"], s["rho"])
    st = dict(kind=kind, E=E)
    if kind == "survey":
        st["shots"] = [swd.ShotSpec(q["sx"], q["sz"], q["rx"], q["rz"], q["nt"]) for q in s["shots"]]
        st["ricks"], st["datas"] = [q["rick"] for q in s["shots"]], [q["data"] for q in s["shots"]]
        return st
    shot = swd.ShotSpec(s["sx"], s["sz"], s["rx"], s["rz"], s["nt"])
    st.update(shot=shot, rick=s["rick"])
    if kind == "rtm":
        E.set_strip_precision(STRIPS[case["strips"]])
        st["data"] = s["data"]
        st["out"] = [torch.zeros(case["nx"], case["nz"], device=DEV) for _ in range(3)]
    elif kind in ("model", "scatter"):
        st.update(hrick=s["hrick"], taper=s["taper"])
        st["out"] = [torch.zeros(len(s["rx"]), s["nt"], device=DEV) for _ in range(3)]
        if kind == "scatter":
            E.set_scatter_model(s["vp"], s["rho1"])
    elif kind == "lsrtm":
        lsrtm = importlib.import_module("swd_b200.lsrtm")
        st["op"] = lsrtm.BornOperator(E, shot, s["rick"], s["vp"].cpu().numpy(), s["rho"].cpu().numpy())
        st["born"] = lsrtm.born
        st["refl"], st["resid"] = s["refl"].requires_grad_(True), s["resid"]
    torch.cuda.synchronize()
    return st


def _check(E, rc):
    if rc != 0:
        raise RuntimeError(_swd().lib().swd_last_error(E._h).decode())


def _p(t):
    return ctypes.c_void_p(t.data_ptr() if hasattr(t, "data_ptr") else t.ctypes.data)


def run(state):
    swd, kind, E = _swd(), state["kind"], state["E"]
    L = swd.lib()
    if kind == "decon":
        c = state["case"]
        if c["host"]:
            w = (c["psfwin"],) * 2, (c["filterwin"],) * 2, (c["snapwin"],) * 2
            return E.decon(state["mig"], state["psf"], *w, EPSILON)
        dec, coef = state["out"]
        _check(E, L.swd_decon(E._h, ctypes.byref(state["prm"]), _p(state["mig"]), _p(state["psf"]), _p(dec), _p(coef)))
        return dec, coef
    if kind == "smooth":
        return E.smooth(state["vp"], state["case"]["pml"] + LC, state["case"]["window"])
    if kind == "survey":
        E.stack_reset()
        E.rtm_batch(state["shots"], state["ricks"], state["datas"])
        return E.stack()
    if kind == "lsrtm":
        d = state["born"](state["refl"], state["op"])
        (g,) = torch.autograd.grad(d, state["refl"], state["resid"])
        return d.detach(), g
    # the remaining calls go through the C interface with arrays on the device
    sh, keep = E._shot(state["shot"])
    a, b, c = state["out"]
    if kind == "rtm":
        _check(E, L.swd_rtm_shot(E._h, ctypes.byref(sh), _p(state["rick"]), _p(state["data"]), swd.RTM_PREPROCESS, None, _p(a), _p(b), _p(c)))
    else:
        f = L.swd_forward if kind == "model" else L.swd_forward_scatter
        _check(E, f(E._h, ctypes.byref(sh), _p(state["rick"]), _p(state["hrick"]), _p(state["taper"]), _p(a), _p(b), _p(c)))
    del keep
    return a, b, c


# ---------------------------------------------------------------------------- work
def work(case):
    """Bytes and operations one pass cannot do without.  Propagation: the model, wavelets and
    records in and the results out, and per step each field of each wavefield read and
    written once with the coefficients read once (the grids do not stay on the chip between
    steps in general); a stencil update of LC taps on both axes is 4 LC + 4 operations."""
    kind = case["kind"]
    if kind == "decon":
        full, out, _, sx, sz = _decon_geometry(case)
        n = full * full
        return {"bytes": 4 * 4 * case["nx"] * case["nz"], "flops": sx * sz * (2 * 5 * n * math.log2(n) + 30 * n)}
    p = case["pml"] + LC
    N, Ni = (case["nx"] + 2 * p) * (case["nz"] + 2 * p), case["nx"] * case["nz"]
    if kind == "smooth":
        w = 2 * case["window"] + 1
        return {"bytes": 8 * N, "flops": 2 * w * w * Ni}
    up = 2 * (4 * LC + 4)   # operations of one cell's velocity and pressure updates
    fwd, bwd = 36 * N, 36 * N + 28 * Ni + 16 * Ni
    if kind == "survey":
        g = 0.75 * case["nt"] * case["shots"]
        return {"bytes": g * (fwd + bwd), "flops": g * (2 * up * N + (up + 4) * Ni)}
    nt, nr = case["nt"], (case["wells"] if case["wells"] == 2 else 0.8) * case["nz"]
    if kind == "rtm":
        return {"bytes": nt * (fwd + bwd) + 4 * nr * nt + 12 * Ni, "flops": nt * (2 * up * N + (up + 4) * Ni)}
    if kind == "model":
        return {"bytes": nt * 60 * N + 12 * nr * nt, "flops": nt * 2 * up * N}
    if kind == "scatter":
        return {"bytes": 2 * nt * 84 * N + 12 * nr * nt, "flops": 2 * nt * 2 * (up + 2) * N}
    return {"bytes": nt * (64 * N + 40 * N + 60 * N) + 8 * nr * nt, "flops": nt * 4 * up * N}   # lsrtm


# ---------------------------------------------------------------------------- exact
class _Fd:
    """The discrete scheme in double precision: staggered velocities and pressure with CPML."""

    def __init__(self, c, s):
        d = lambda a: torch.as_tensor(a, device=DEV).double()
        self.nt, self.dt, self.p0 = c["nt"], float(np.float32(c["dt"])), c["pml"] + LC
        self.h = float(np.float32(c["h"]))
        self.rc = [float(v) / self.h for v in s["rc"]]
        self.vp, self.rho = s["vp"].double(), s["rho"].double()
        self.X, self.Z = self.vp.shape
        self.nx, self.nz = c["nx"], c["nz"]
        q = {k: d(v) for k, v in s["cpml"].items()}
        n, m = self.X - 2 * LC + 1, self.Z - 2 * LC + 1
        self.n, self.m = n, m
        lo, hi = slice(LC - 1, LC - 1 + n), slice(LC, LC + n)
        zl, zh = slice(LC - 1, LC - 1 + m), slice(LC, LC + m)
        self.lo, self.hi, self.zl, self.zh = lo, hi, zl, zh
        self.axh, self.bxh = q["a_x_half"][lo, None], q["b_x_half"][lo, None]
        self.ax, self.bx = q["a_x"][hi, None], q["b_x"][hi, None]
        self.azh, self.bzh = q["a_z_half"][None, zl], q["b_z_half"][None, zl]
        self.az, self.bz = q["a_z"][None, zh], q["b_z"][None, zh]
        self.coefs(self.vp, self.rho)

    def coefs(self, vp, rho):
        self.cbx = self.dt / (0.5 * (rho[:-1] + rho[1:]))[self.lo]
        self.cbz = self.dt / (0.5 * (rho[:, :-1] + rho[:, 1:]))[:, self.zl]
        self.kap = rho * vp * vp
        self.ck = self.dt * self.kap

    def dx(self, f):
        o = None
        for i, c in enumerate(self.rc):
            t = f[LC + i:LC + i + self.n] - f[LC - 1 - i:LC - 1 - i + self.n]
            o = t.mul_(c) if o is None else o.add_(t, alpha=c)
        return o

    def dz(self, f):
        o = None
        for i, c in enumerate(self.rc):
            t = f[:, LC + i:LC + i + self.m] - f[:, LC - 1 - i:LC - 1 - i + self.m]
            o = t.mul_(c) if o is None else o.add_(t, alpha=c)
        return o

    def dxt(self, g, out):
        for i, c in enumerate(self.rc):
            out[LC + i:LC + i + self.n].add_(g, alpha=c)
            out[LC - 1 - i:LC - 1 - i + self.n].add_(g, alpha=-c)

    def dzt(self, g, out):
        for i, c in enumerate(self.rc):
            out[:, LC + i:LC + i + self.m].add_(g, alpha=c)
            out[:, LC - 1 - i:LC - 1 - i + self.m].add_(g, alpha=-c)

    def zero(self):
        z = lambda a, b: torch.zeros(a, b, device=DEV, dtype=torch.float64)
        return dict(p=z(self.X, self.Z), vx=z(self.X, self.Z), vz=z(self.X, self.Z), ppx=z(self.n, self.Z),
                    ppz=z(self.X, self.m), pvx=z(self.n, self.m), pvz=z(self.n, self.m))

    def v(self, w, sign=1.0, wide=False):
        """Velocity half step; the receiver wavefield runs with negated spacing and wide guards."""
        rows = slice(0, self.Z) if wide else self.zh
        cols = slice(0, self.X) if wide else self.hi
        d = self.dx(w["p"])[:, rows] * sign
        f = w["ppx"][:, rows]
        f.mul_(self.bxh).add_(self.axh * d)
        w["vx"][self.lo, rows] += self.cbx[:, rows] * (d + f)
        d = self.dz(w["p"])[cols] * sign
        f = w["ppz"][cols]
        f.mul_(self.bzh).add_(self.azh * d)
        w["vz"][cols, self.zl] += self.cbz[cols] * (d + f)

    def p(self, w, sign=1.0):
        d = self.dx(w["vx"])[:, self.zh] * sign
        w["pvx"].mul_(self.bx).add_(self.ax * d)
        s = d + w["pvx"]
        d = self.dz(w["vz"])[self.hi] * sign
        w["pvz"].mul_(self.bz).add_(self.az * d)
        s = s + d + w["pvz"]
        w["p"][self.hi, self.zh] += self.ck[self.hi, self.zh] * s
        return s

    def band(self):
        """Indices of the boundary band of width LC inside the interior's edge."""
        m = torch.zeros(self.X, self.Z, device=DEV, dtype=torch.bool)
        a, b, e, f = self.p0, self.X - self.p0, self.p0, self.Z - self.p0
        m[a:b, e:f] = True
        m[a + LC:b - LC, e + LC:f - LC] = False
        return m.reshape(-1).nonzero().reshape(-1)


def _exact_shot(fd, sx, sz, rx, rz, nt, rick, data):
    """Filtered image, illumination and normalised image of one shot."""
    rick = [float(v) for v in rick]
    rx, rz = (torch.as_tensor(a, device=DEV).long() for a in (rx, rz))
    w, idx = fd.zero(), fd.band()
    strips = torch.empty(nt, len(idx), device=DEV, dtype=torch.float64)
    for it in range(nt):
        fd.v(w)
        fd.p(w)
        w["p"][sx, sz] += rick[it]
        strips[it] = w["p"].reshape(-1)[idx]
    rms = -torch.cumsum(torch.cumsum(data.double() * fd.dt, 1) * fd.dt, 1)
    r = fd.zero()
    I, S = torch.zeros_like(w["p"]), torch.zeros_like(w["p"])
    a, b, e, f = fd.p0, fd.X - fd.p0, fd.p0, fd.Z - fd.p0
    ox, oz = fd.p0 - LC, fd.p0 - LC   # interior within the dx / dz output (origin LC for p, LC - 1 for v)
    for it in range(nt - 2, -1, -1):
        s = fd.dx(w["vx"])[ox:ox + fd.nx, e:f] + fd.dz(w["vz"])[a:b, oz:oz + fd.nz]
        w["p"][a:b, e:f] -= fd.ck[a:b, e:f] * s
        dp = fd.kap[a:b, e:f] * s
        w["p"][sx, sz] -= rick[it + 1]
        w["p"].reshape(-1)[idx] = strips[it]
        w["vx"][a:b, e:f] -= fd.cbx[ox + 1:ox + 1 + fd.nx, e:f] * fd.dx(w["p"])[ox + 1:ox + 1 + fd.nx, e:f]
        w["vz"][a:b, e:f] -= fd.cbz[a:b, oz + 1:oz + 1 + fd.nz] * fd.dz(w["p"])[a:b, oz + 1:oz + 1 + fd.nz]
        fd.v(r, -1.0, True)
        fd.p(r, -1.0)
        r["p"][rx, rz] = rms[:, it]
        I[a:b, e:f] += dp * r["p"][a:b, e:f]
        S[a:b, e:f] += dp * dp
    In = I / (S + 1.0e-3 * S.max())
    h2 = fd.h * fd.h
    lap = (In[a + 1:b + 1, e:f] + In[a - 1:b - 1, e:f] + In[a:b, e + 1:f + 1] + In[a:b, e - 1:f - 1] - 4.0 * In[a:b, e:f]) / h2
    return In[a:b, e:f], S[a:b, e:f], -lap * fd.vp[a:b, e:f] ** 2


def _exact_split(cols, taper, rz):
    """Up- and down-going traces of recorded complex columns (nt, Z)."""
    n = len(taper)
    f = torch.fft.fft(cols, n, dim=1) * torch.as_tensor(taper, device=DEV).double()
    up = f.clone()
    up[:, n // 2 + 1:] = 0.0
    out = []
    for q in (up, f - up):
        out.append((torch.fft.ifft(q, dim=1).real * n)[:, rz].T.contiguous())
    return out


def _exact_records(fd, s, model=None):
    """Record of one modelling run and its up/down parts, from the wavelet and its Hilbert twin."""
    rx, rz = (torch.as_tensor(a, device=DEV).long() for a in (s["rx"], s["rz"]))
    xs = sorted(set(s["rx"].tolist()))
    cols = {x: torch.zeros(s["nt"], fd.Z, device=DEV, dtype=torch.complex128) for x in xs}
    for part, wav in ((0, s["rick"]), (1, s["hrick"])):
        w = fd.zero()
        for it in range(s["nt"]):
            fd.v(w)
            fd.p(w)
            w["p"][s["sx"], s["sz"]] += float(wav[it])
            for x in xs:
                (cols[x].real if part == 0 else cols[x].imag)[it] = w["p"][x]
    seis = torch.stack([cols[int(x)].real[:, int(z)] for x, z in zip(s["rx"], s["rz"])])
    return seis, cols


def _exact_decon(case, seed):
    mig, psf = (a.double() for a in _decon_inputs(case, seed))
    nx, nz, w, fw, sn = case["nx"], case["nz"], case["psfwin"], case["filterwin"], case["snapwin"]
    full, out, step, sx, sz = _decon_geometry(case)
    hp, hf, ho, mid = w // 2, fw // 2, out // 2, full // 2
    nxp, nzp, lx, lz = sx * step, sz * step, math.ceil(nx / w), math.ceil(nz / w)
    ar = lambda n: torch.arange(n, device=DEV)
    k = np.arange(out)
    t = np.where(k < sn, 0.5 - 0.5 * np.cos(3.1415926 * k / (sn - 1)), np.where(k >= out - sn, 0.5 + 0.5 * np.cos(3.1415926 * (k - out + sn) / (sn - 1)), 1.0))
    t = torch.as_tensor(t, device=DEV)
    taper = t[:, None] * t[None, :]
    dec = torch.zeros(nxp + 2 * out, nzp + 2 * out, device=DEV, dtype=torch.float64)
    coef = torch.zeros_like(dec)
    eps = float(np.float32(EPSILON))
    for a in range(sx):
        ix = torch.tensor([a * step], device=DEV)
        iz = ar(sz) * step
        def lattice(i, n):
            f = torch.div(i - hp, w, rounding_mode="trunc")
            f = torch.where(f <= 2, 3, f)
            return hp + torch.where(f >= n - 3, n - 4, f) * w
        px, pz = lattice(ix, lx), lattice(iz, lz)
        gx, gz = ix[:, None] - hf + ar(fw), iz[:, None] - hf + ar(fw)
        ok = ((gx >= 0) & (gx < nxp))[:, :, None] & ((gz >= 0) & (gz < nzp))[:, None, :]
        M = mig[gx.clamp(0, nx - 1)[:, :, None], gz.clamp(0, nz - 1)[:, None, :]] * ok
        P = psf[(px[:, None] - hp + ar(w)).clamp(0, nx - 1)[:, :, None], (pz[:, None] - hp + ar(w)).clamp(0, nz - 1)[:, None, :]].expand(sz, w, w)
        m1 = M.abs().sum((1, 2), keepdim=True)
        m1 = torch.where(m1 <= 1.0e-15, torch.full_like(m1, 1.0e-10), m1)
        B = torch.zeros(sz, full, full, device=DEV, dtype=torch.float64)
        B[:, mid - hf:mid - hf + fw, mid - hf:mid - hf + fw] = M / m1
        Q = torch.zeros_like(B)
        Q[:, :w, :w] = P / P.abs().sum((1, 2), keepdim=True)
        FM, FQ = torch.fft.fft2(B), torch.fft.fft2(Q)
        pw = FQ.real ** 2 + FQ.imag ** 2
        damp = eps * pw.amax((1, 2), keepdim=True)
        damp = torch.where(damp == 0.0, torch.full_like(damp, 1.0e-15), damp)
        D = torch.fft.ifft2(FM * FQ.conj() / (pw + damp)).real * (full * full)
        oc = mid - hp - ho
        D = D[:, oc:oc + out, oc:oc + out] * taper
        x0 = a * step - ho + out
        for b in range(sz):
            z0 = b * step - ho + out
            dec[x0:x0 + out, z0:z0 + out] += D[b]
            coef[x0:x0 + out, z0:z0 + out] += taper
    return dec[out:out + nx, out:out + nz].contiguous(), coef[out:out + nx, out:out + nz].contiguous()


def _exact_smooth(case, seed):
    p, w = case["pml"] + LC, case["window"]
    v = _pad(_velocity(case["nx"], case["nz"], _gen(seed)), p).double()
    i = torch.arange(-w, w + 1, device=DEV, dtype=torch.float64)
    k = torch.exp(-(i * i) / (2.0 * (w / 2.0) ** 2))
    k = k / k.sum()
    s = torch.nn.functional.pad(v[None, None], (w, w, w, w), mode="replicate")[0, 0]
    s = sum(k[j] * s[j:j + v.shape[0]] for j in range(2 * w + 1))
    s = sum(k[j] * s[:, j:j + v.shape[1]] for j in range(2 * w + 1))
    s = s[p:-p, p:-p].clone()
    s[:, :8] = v[p:-p, p:p + 8]
    return torch.nn.functional.pad(s[None, None], (p, p, p, p), mode="replicate")[0, 0].contiguous().cpu()


def exact(case, seed):
    kind = case["kind"]
    if kind == "decon":
        out = _exact_decon(case, seed)
        return tuple(a.cpu() for a in out) if case["host"] else out
    if kind == "smooth":
        return _exact_smooth(case, seed)
    s = _grid_inputs(case, seed)
    fd = _Fd(case, s)
    if kind == "rtm":
        return _exact_shot(fd, s["sx"], s["sz"], s["rx"], s["rz"], s["nt"], s["rick"], s["data"])
    if kind == "survey":
        st = 0.0
        for q in s["shots"]:
            st = st + _exact_shot(fd, q["sx"], q["sz"], q["rx"], q["rz"], q["nt"], q["rick"], q["data"])[2]
        st[:4], st[fd.nx - LC:], st[:, :7], st[:, fd.nz - LC:] = 0.0, 0.0, 0.0, 0.0
        return st.cpu()
    if kind in ("model", "scatter"):
        seis, cols = _exact_records(fd, s)
        if kind == "scatter":   # difference of two runs, the perturbed model less the background
            fd.coefs(fd.vp, s["rho1"].double())
            seis1, cols1 = _exact_records(fd, s)
            seis, cols = seis1 - seis, {x: cols1[x] - cols[x] for x in cols}
        up, dn = torch.empty_like(seis), torch.empty_like(seis)
        for x in cols:
            here = torch.as_tensor(s["rx"] == x, device=DEV)
            u, d = _exact_split(cols[x], s["taper"], torch.as_tensor(s["rz"][s["rx"] == x], device=DEV).long())
            up[here], dn[here] = u, d
        return seis, up, dn
    # lsrtm: Born data and the transpose of that linear map applied to the residual
    rx, rz = (torch.as_tensor(a, device=DEV).long() for a in (s["rx"], s["rz"]))
    p, nt = fd.p0, s["nt"]
    inner = (slice(p, p + fd.nx), slice(p, p + fd.nz))
    dk = torch.zeros_like(fd.vp)
    dk[inner] = 2.0 * fd.kap[inner] * s["refl"].double()
    w, u = fd.zero(), fd.zero()
    S0 = torch.empty(nt, fd.n, fd.m, device=DEV, dtype=torch.float64)
    d = torch.empty(nt, len(rx), device=DEV, dtype=torch.float64)
    for it in range(nt):
        fd.v(w)
        fd.v(u)
        S0[it] = fd.p(w)
        fd.p(u)
        u["p"][fd.hi, fd.zh] += fd.dt * dk[fd.hi, fd.zh] * S0[it]
        w["p"][s["sx"], s["sz"]] += float(s["rick"][it])
        d[it] = u["p"][rx, rz]
    del w, u
    l = fd.zero()
    g = torch.zeros(fd.n, fd.m, device=DEV, dtype=torch.float64)
    res = s["resid"].double()
    for it in range(nt - 1, -1, -1):
        l["p"].index_put_((rx, rz), res[:, it], accumulate=True)
        lp = l["p"][fd.hi, fd.zh]
        g += fd.dt * S0[it] * lp
        q = fd.ck[fd.hi, fd.zh] * lp
        for f, a, b, t in (("pvx", fd.ax, fd.bx, 0), ("pvz", fd.az, fd.bz, 1)):
            gp = l[f] + q
            e = q + a * gp
            l[f] = b * gp
            if t == 0:
                full = torch.zeros(fd.n, fd.Z, device=DEV, dtype=torch.float64)
                full[:, fd.zh] = e
                fd.dxt(full, l["vx"])
            else:
                full = torch.zeros(fd.X, fd.m, device=DEV, dtype=torch.float64)
                full[fd.hi] = e
                fd.dzt(full, l["vz"])
        r = fd.cbx[:, fd.zh] * l["vx"][fd.lo, fd.zh]
        gp = l["ppx"][:, fd.zh] + r
        e = torch.zeros(fd.n, fd.Z, device=DEV, dtype=torch.float64)
        e[:, fd.zh] = r + fd.axh * gp
        l["ppx"][:, fd.zh] = fd.bxh * gp
        r = fd.cbz[fd.hi] * l["vz"][fd.hi, fd.zl]
        gp = l["ppz"][fd.hi] + r
        ez = torch.zeros(fd.X, fd.m, device=DEV, dtype=torch.float64)
        ez[fd.hi] = r + fd.azh * gp
        l["ppz"][fd.hi] = fd.bzh * gp
        fd.dxt(e, l["p"])
        fd.dzt(ez, l["p"])
    full = torch.zeros_like(fd.vp)
    full[fd.hi, fd.zh] = g
    return d.T.contiguous(), 2.0 * fd.kap[inner] * full[inner]
