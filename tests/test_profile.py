"""Profiling times the kernels that run without it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (nx, nz, pml, nt): a grid whose passes stay on the chip, one whose forward steps march, one between
CASES = {"chip": (100, 60, 10, 130), "march": (3001, 1509, 13, 140), "steps": (1201, 601, 10, 140)}


@pytest.mark.parametrize("name", list(CASES))
def test_profiled_passes_launch_the_same_kernels(swd, name):
    nx, nz, pml, nt = CASES[name]
    p = pml + 4
    E = swd.Engine(nx, nz, pml, 4, 5.0, 5.0, 5e-4, nt)
    vp = np.full((nx + 2 * p, nz + 2 * p), 2000.0, np.float32)
    E.setup_default(vp, np.full_like(vp, 1000.0))
    s = swd.ShotSpec(p + 20, p + 4, np.full(9, p + 30, np.int32), (p + np.arange(9)).astype(np.int32), nt)
    rick = swd.ricker_wave(nt, 40.0, 5e-4)
    data = np.ones((9, nt), np.float32)
    out, count = [], []
    for every in (0, 8):
        E.profile(every)
        n0 = E.launch_count()
        E.rtm_shot(s, rick, data, flags=swd.RTM_NO_STACK, want=())
        out.append(E.rtm_raw()[:2])
        count.append(E.launch_count() - n0)
    prof = E.profile_read()
    assert count[0] == count[1]
    for a, b in zip(*out):
        assert np.abs(a).max() > 0 and np.array_equal(a, b)
    assert prof["fwd_pass_step"][1] == nt and prof["bwd_pass_step"][1] == nt - 1
    for k in ("fwd_pass_step", "bwd_pass_step"):
        assert prof[k][0] > 0
    one = {"chip": ("fwd_step", "bwd_step"), "march": ("fwd_step", "bwd_1", "bwd_2"), "steps": ("fwd_v", "fwd_p", "bwd_1", "bwd_2")}[name]
    assert {k for k in ("fwd_v", "fwd_p", "bwd_1", "bwd_2", "fwd_step", "bwd_step") if prof[k][1]} == set(one)
