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


class Rtm:
    """One shot on a grid whose forward pass takes a second copy of the field (94 MB)."""

    nt = 66

    def __init__(self, swd):
        nx, nz, pml = 3001, 1509, 13
        rng = np.random.default_rng(3)
        self.swd, p = swd, pml + 4
        self.vp = swd.pad_model((1900.0 + 900.0 * np.arange(nz)[None, :] / nz + rng.uniform(-80, 80, (nx, 1))).astype(np.float32), p)
        self.rho = np.full_like(self.vp, 1000.0)
        self.dims = (nx, nz, pml, 4, 5.0, 5.0, 5e-4, self.nt)
        self.shot = swd.ShotSpec(p + nx // 2, p + 4, np.full(40, p + nx // 2 + 5, np.int32), (p + np.arange(40)).astype(np.int32), self.nt)
        self.rick = swd.ricker_wave(self.nt, 60.0, 5e-4)
        self.data = rng.standard_normal((40, self.nt)).astype(np.float32)

    def engine(self):
        E = self.swd.Engine(*self.dims)
        E.setup_default(self.vp, self.rho)
        return E

    def backward(self, E):
        E.rtm_backward(self.shot, self.data, flags=self.swd.RTM_NO_STACK, want=())
        return E.rtm_raw()[:2]

    def steps(self, E):
        """The shot by the step kernels (no second copy)."""
        E.set_option(self.swd.OPT_MARCH, 0)
        E.rtm_forward(self.shot, self.rick)
        return self.backward(E)


@pytest.mark.parametrize("first", ["march", "smooth", "decon"])
def test_scratch_of_an_earlier_call_is_given_back(swd, first):
    """The second call needs more than is left on the device, but no more than with the scratch of the
    first (94 to 160 MB) given back."""
    job = Rtm(swd)
    other = Decon(swd) if first == "decon" else None
    big = np.full((5000, 4000), 2000.0, np.float32)

    def begin(E):
        if first == "march":
            E.rtm_forward(job.shot, job.rick)
        elif first == "smooth":
            E.smooth(big, 17, 2)
        else:
            other(E)

    end = job.backward if first == "march" else job.steps
    E = job.engine()
    begin(E)
    n0 = E.device_bytes()
    ref = end(E)
    need = E.device_bytes() - n0
    E.close()
    E = job.engine()
    begin(E)
    with Filled(need - 20 * MB):
        got = end(E)
    for a, b in zip(got, ref):
        assert np.abs(b).max() > 0 and np.array_equal(a, b)


def test_march_without_room_for_its_second_copy(swd):
    job = Rtm(swd)
    E = job.engine()
    E.set_option(swd.OPT_MARCH, 0)
    n0 = E.device_bytes()
    ref = E.forward(job.shot, job.rick)
    need = E.device_bytes() - n0
    E.close()
    E = job.engine()
    with Filled(need + 45 * MB):
        n0 = E.launch_count()
        got = E.forward(job.shot, job.rick)
        assert E.launch_count() - n0 >= 2 * job.nt
    assert np.abs(ref).max() > 0 and np.array_equal(got, ref)
    n0 = E.launch_count()
    assert np.array_equal(E.forward(job.shot, job.rick), ref)
    assert E.launch_count() - n0 < 2 * job.nt


def test_on_chip_pass_without_room_for_its_exchange_words(swd):
    """Every buffer of the step kernels is there, and not two megabytes more."""
    drv = C.CDLL("libcuda.so.1")
    nt = 60
    E = swd.Engine(401, 201, 10, 4, 5.0, 5.0, 5e-4, nt)
    vp = np.full((429, 229), 2000.0, np.float32)
    E.setup_default(vp, np.full_like(vp, 1000.0))
    s = swd.ShotSpec(60, 16, np.full(20, 70, np.int32), np.arange(20, 40).astype(np.int32), nt)
    rick = swd.ricker_wave(nt, 60.0, 5e-4)
    E.set_option(swd.OPT_RESIDENT, 0)
    ref = E.forward(s, rick)
    E.set_option(swd.OPT_RESIDENT, 1)
    taken = []
    with Filled(64 * MB):
        for n in (16, 8, 4, 2):
            p = C.c_uint64()
            while len(taken) < 100 and drv.cuMemAlloc_v2(C.byref(p), C.c_size_t(n * MB)) == 0:
                taken.append(p.value)
        got = E.forward(s, rick)
        for p in taken:
            assert drv.cuMemFree_v2(C.c_uint64(p)) == 0
    assert np.abs(ref).max() > 0 and np.array_equal(got, ref)
    n0 = E.launch_count()
    assert np.array_equal(E.forward(s, rick), ref)
    assert E.launch_count() - n0 < nt                   # on the chip again


def test_decon_without_a_context_frees_what_it_took(swd):
    """The same result as with a context, arrays on the device and on the host, and no memory kept; on a
    nearly full device by the FFT windows."""
    job = Decon(swd)
    none = type("NoContext", (), {"_h": None, "_ck": staticmethod(lambda rc: rc == 0 or pytest.fail(f"error {rc}"))})
    E = swd.Engine(64, 64, 8, 4, 5.0, 5.0, 5e-4, 64)
    ref = job(E)
    E.close()
    job(none)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    assert np.array_equal(job(none), ref)
    with Filled(152 * MB):
        assert rel_l2(job(none), ref) < 2e-5
    host = swd.decon(*[t.cpu().numpy() for t in job.ins], (79, 79), (79, 79), (24, 24), 1e-3, psf_interp=1)[0]
    assert np.array_equal(host, ref)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free
