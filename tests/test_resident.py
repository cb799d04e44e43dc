"""On-chip time loops (SWD_OPT_RESIDENT) against the step kernels: the same bits.

The grids sit where the tiling can go wrong: one row or one column in the last tile, exactly full
tiles, one tile only along z, the smallest grid, one and two columns per warp at the ends of their
ranges, the largest grid that fits; receivers scattered over the whole padded grid (several per
warp and per cell column, duplicates, frame cells), the source inside the strip band and in the
frame.  The arithmetic is the same term by term, so the comparison is exact."""
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest
import torch

from conftest import ROOT

pytestmark = pytest.mark.gpu

# (nx, nz, pml): padded sizes are nx + 2 * (pml + 4)
GRIDS = {
    "smallest": (20, 20, 10),              # 48 x 48, one tile row, 8-column tiles
    "z_full_tile": (100, 100, 10),         # 128 rows: exactly one tile
    "z_one_row_left": (101, 101, 10),      # 129 x 129: last tile one row, last column tile one column
    "x_13_columns": (620, 300, 10),        # 648 x 328: 13-column tiles, one column per warp, 16-warp kernel
    "x_17_columns": (600, 400, 10),        # 628 x 428: two columns per warp, shortest
    "x_24_columns": (850, 400, 15),        # 888 x 438: 24-column tiles, full
}


def _engine(swd, nx, nz, pml, nt, seed):
    rng = np.random.default_rng(seed)
    pmlc = pml + 4
    v = (1900.0 + 900.0 * np.arange(nz)[None, :] / nz + rng.uniform(-80, 80, (nx, nz))).astype(np.float32)
    vp = swd.pad_model(v, pmlc)
    rho = (1000.0 + rng.uniform(-50, 50, vp.shape)).astype(np.float32)
    E = swd.Engine(nx, nz, pml, 4, 5.0, 5.0, 5e-4, nt)
    E.setup_default(vp, rho)
    return E, rng, vp.shape


@pytest.mark.parametrize("name", list(GRIDS))
def test_resident_same_bits(swd, name):
    nx, nz, pml = GRIDS[name]
    nt = 150
    E, rng, (ntx, ntz) = _engine(swd, nx, nz, pml, nt, 5)
    pmlc = pml + 4
    n = 60
    rix, riz = rng.integers(0, ntx, n).astype(np.int32), rng.integers(0, ntz, n).astype(np.int32)
    rix[:20] = pmlc + nx // 2          # a well, with two traces on one cell
    riz[:20] = np.minimum(pmlc + np.arange(20), ntz - 1)
    riz[1] = riz[0]
    rick = swd.ricker_wave(nt, 25.0, 5e-4)
    hr = E.hilbert(rick)
    coef = rng.uniform(0.2, 1.0, swd.pow2(ntz)).astype(np.float32)
    data = rng.standard_normal((n, nt)).astype(np.float32)
    out = {}
    for res in (0, 1):
        E.set_option(swd.OPT_RESIDENT, res)
        r = []
        n0 = E.launch_count()
        for sx, sz in ((pmlc + nx // 2, pmlc + 1), (3, ntz - 5)):
            s = swd.ShotSpec(sx, sz, rix, riz, nt)
            r.append(E.forward(s, rick))
            r += list(E.forward(s, rick, hrick=hr, kz_coef=coef))
            o = E.rtm_shot(s, rick, data, flags=swd.RTM_PREPROCESS | swd.RTM_NO_STACK, want=("image_pp", "image_src", "fimage", "syn"))
            r += [o[k] for k in sorted(o)] + list(E.rtm_raw()[:2])
            E.stack_reset()
            E.rtm_batch([s, swd.ShotSpec(sx, sz, rix, riz, nt - 37)], [rick, rick[:nt - 37]], [data, data[:, :nt - 37].copy()])
            r.append(E.stack(edge_zero=False))
        out[res] = (r, E.launch_count() - n0)
    assert E.get_option(swd.OPT_RESIDENT) == 1          # no pass gave up
    assert out[1][1] < 0.1 * out[0][1]                  # and the time loops really ran as single launches
    for i, (a, b) in enumerate(zip(out[1][0], out[0][0])):
        assert i >= len(out[0][0]) // 2 or np.abs(b).max() > 0, i   # (the corner source is too far from some receivers)
        assert np.array_equal(a, b), i


def test_resident_needs_its_sizes(swd):
    """A grid too large for the chip, another stencil length and 16-bit strips keep the step kernels."""
    for nx, nz, Lc, prec in ((1200, 600, 4, 0), (100, 60, 3, 0), (100, 60, 4, 1)):
        nt = 64
        E = swd.Engine(nx, nz, 10, Lc, 5.0, 5.0, 5e-4, nt)
        vp = np.full((nx + 2 * (10 + Lc), nz + 2 * (10 + Lc)), 2000.0, np.float32)
        E.setup_default(vp, np.full_like(vp, 1000.0))
        E.set_strip_precision(prec)
        s = swd.ShotSpec(30, 30, np.array([40], np.int32), np.array([30], np.int32), nt)
        n0 = E.launch_count()
        E.rtm_forward(s, swd.ricker_wave(nt, 25.0, 5e-4))
        assert E.launch_count() - n0 >= 2 * nt


@pytest.mark.parametrize("name", list(GRIDS))
def test_resident_born_same_bits(swd, name):
    """Born modelling and the recomputed background of its adjoint, in pieces of the checkpoint
    interval: full storage, the shortest piece taken, a last piece of one step, one piece only, and
    an interval below the shortest piece; checkpoints of 32 and of 16 bits."""
    nx, nz, pml = GRIDS[name]
    nt = 121
    E, rng, (ntx, ntz) = _engine(swd, nx, nz, pml, nt, 7)
    pmlc = pml + 4
    n = 40
    rix, riz = rng.integers(0, ntx, n).astype(np.int32), rng.integers(0, ntz, n).astype(np.int32)
    rix[:20] = pmlc + nx // 2
    riz[:20] = np.minimum(pmlc + np.arange(20), ntz - 1)
    riz[1] = riz[0]
    rick = swd.ricker_wave(nt, 25.0, 5e-4)
    s = swd.ShotSpec(pmlc + nx // 2, pmlc + 1, rix, riz, nt)
    dk = (rng.standard_normal((ntx, ntz)) * 1e7).astype(np.float32)
    resid = rng.standard_normal((n, nt)).astype(np.float32)
    out = {}
    for res in (0, 1):
        E.set_option(swd.OPT_RESIDENT, res)
        r = []
        for every, prec in ((0, swd.STRIP_F32), (8, swd.STRIP_F32), (40, swd.STRIP_BF16), (500, swd.STRIP_I16), (7, swd.STRIP_F16)):
            E.set_checkpointing(every, prec)
            ck = torch.empty(max(16, E.checkpoint_bytes(nt)), dtype=torch.uint8, device="cuda") if every else None
            n0 = E.launch_count()
            r.append(E.born(s, rick, dk, ckpt=ck))
            assert E.launch_count() - n0 >= 2 * nt if not res or 0 < every < 8 else E.launch_count() - n0 < nt
            r += [E.born_adjoint(s, rick, resid, ckpt=ck), E.born_adjoint(s, rick, resid)]
        out[res] = r
    assert E.get_option(swd.OPT_RESIDENT) == 1
    for i, (a, b) in enumerate(zip(out[1], out[0])):
        assert np.abs(b).max() > 0, i
        assert np.array_equal(a, b), i


def test_engines_side_by_side_same_bits(swd):
    """Engines that run at the same time (their calls choose the step kernels while another call is in
    progress) give what one engine gives alone."""
    nt = 150
    made = [_engine(swd, 100, 100, 10, nt, 3) for _ in range(3)]
    ntx, ntz = made[0][2]
    rng = np.random.default_rng(8)
    s = swd.ShotSpec(60, 20, np.full(40, 70, np.int32), np.arange(20, 60).astype(np.int32), nt)
    rick, data = swd.ricker_wave(nt, 25.0, 5e-4), rng.standard_normal((40, nt)).astype(np.float32)

    def shots(E, n):
        r = []
        for _ in range(n):
            E.rtm_shot(s, rick, data, flags=swd.RTM_NO_STACK, want=())
            r += [E.forward(s, rick)] + list(E.rtm_raw()[:2])
        return r

    ref = shots(made[0][0], 1)
    with ThreadPoolExecutor(3) as pool:
        out = list(pool.map(lambda m: shots(m[0], 6), made))
    for r in out:
        for k, a in enumerate(r):
            assert np.array_equal(a, ref[k % 3])


@pytest.mark.parametrize("nz,pml", [(9, 30), (9, 17), (10, 17), (11, 17)])
def test_models_of_few_rows_same_bits(swd, nz, pml):
    """Models whose top and bottom strips lie within four rows of each other."""
    nt = 120
    E, rng, (ntx, ntz) = _engine(swd, 60, nz, pml, nt, 4)
    pmlc = pml + 4
    rix, riz = np.full(nz, pmlc + 40, np.int32), (pmlc + np.arange(nz)).astype(np.int32)
    s = swd.ShotSpec(pmlc + 20, pmlc + 4, rix, riz, nt)
    rick, data = swd.ricker_wave(nt, 25.0, 5e-4), rng.standard_normal((nz, nt)).astype(np.float32)
    out = []
    for res in (0, 1):
        E.set_option(swd.OPT_RESIDENT, res)
        r = E.rtm_shot(s, rick, data, flags=swd.RTM_NO_STACK)
        out.append([r[k] for k in sorted(r)] + list(E.rtm_raw()[:2]))
    for a, b in zip(*out):
        assert np.abs(b).max() > 0
        assert np.array_equal(a, b)


GIVE_UP = ["forward", "twin", "rtm_shot", "rtm_forward", "rtm_backward", "batch", "born", "born_checkpoints", "adjoint", "adjoint_checkpoints"]


def _gives_up(swd, grid, name, stops, nt=60):
    """The call `name` by the step kernels, then on the chip with each SWD_OPT_RESIDENT_STOP in turn, then
    undisturbed: the same bits (results and stack) every time, and the option reads 0 after a pass that
    gave up."""
    nx, nz, pml = GRIDS[grid]
    E, rng, (ntx, ntz) = _engine(swd, nx, nz, pml, nt, 6)
    pmlc = pml + 4
    rix, riz = np.full(20, pmlc + nx // 2, np.int32), (pmlc + np.arange(20)).astype(np.int32)
    s = swd.ShotSpec(pmlc + nx // 2 - 6, pmlc + 1, rix, riz, nt)
    rick = swd.ricker_wave(nt, 60.0, 5e-4)
    hr, coef = E.hilbert(rick), rng.uniform(0.2, 1.0, swd.pow2(ntz)).astype(np.float32)
    data = rng.standard_normal((20, nt)).astype(np.float32)
    dk = (rng.standard_normal((ntx, ntz)) * 1e7).astype(np.float32)
    E.set_checkpointing(16 if name.endswith("checkpoints") else 0, swd.STRIP_F32)
    ck = torch.empty(max(16, E.checkpoint_bytes(nt)), dtype=torch.uint8, device="cuda") if name.endswith("checkpoints") else None

    def call(stop):
        E.stack_reset()
        E.set_option(swd.OPT_RESIDENT_STOP, 0 if name == "rtm_backward" else stop)
        if name == "forward":
            return [E.forward(s, rick)]
        if name == "twin":
            return list(E.forward(s, rick, hrick=hr, kz_coef=coef))
        if name == "rtm_shot":
            o = E.rtm_shot(s, rick, data, want=("image_pp", "image_src", "fimage", "syn"))
            return [o[k] for k in sorted(o)] + list(E.rtm_raw()[:2]) + [E.stack(edge_zero=False)]
        if name == "rtm_forward":
            r = [E.rtm_forward(s, rick, syn=True)]
            E.set_option(swd.OPT_RESIDENT_STOP, 0)
            E.rtm_backward(s, data, want=())
            return r + list(E.rtm_raw()[:2]) + [E.stack(edge_zero=False)]
        if name == "rtm_backward":
            E.rtm_forward(s, rick)
            E.set_option(swd.OPT_RESIDENT_STOP, stop)
            o = E.rtm_backward(s, data)
            return [o[k] for k in sorted(o)] + list(E.rtm_raw()[:2]) + [E.stack(edge_zero=False)]
        if name == "batch":
            E.rtm_batch([s, s], [rick, rick], [data, 2 * data])
            return [E.stack(edge_zero=False)]
        if name.startswith("born"):
            return [E.born(s, rick, dk, ckpt=ck)] + ([E.born_adjoint(s, rick, data, ckpt=ck)] if ck is not None else [])
        if ck is not None:
            E.set_option(swd.OPT_RESIDENT_STOP, 0)
            E.born(s, rick, dk, ckpt=ck)
            E.set_option(swd.OPT_RESIDENT_STOP, stop)
        return [E.born_adjoint(s, rick, data, ckpt=ck)]

    E.set_option(swd.OPT_RESIDENT, 0)
    ref = call(0)
    for stop in list(stops) + [0]:
        E.set_option(swd.OPT_RESIDENT, 1)
        got = call(stop)
        assert E.get_option(swd.OPT_RESIDENT) == (1 if stop == 0 else 0)
        for i, (a, b) in enumerate(zip(got, ref)):
            assert np.abs(b).max() > 0, (stop, i)
            assert np.array_equal(a, b), (stop, i)


@pytest.mark.parametrize("name", GIVE_UP)
@pytest.mark.parametrize("grid", ["z_one_row_left", "x_24_columns"])
def test_pass_that_gives_up_runs_again(swd, grid, name):
    """Passes that stop after their first step and after some: the call runs again
    with the step kernels, and a later pass on the chip is not disturbed by the stopped one."""
    _gives_up(swd, grid, name, (1, 13))


@pytest.mark.parametrize("name", ["rtm_shot", "adjoint_checkpoints"])
def test_waits_that_run_out(swd, name):
    """One tile does not start: its neighbours wait for its words until their tries run out, and theirs
    in turn."""
    _gives_up(swd, "smallest", name, (-1,))


@pytest.mark.parametrize("name", GIVE_UP)
def test_refused_launch_runs_the_step_kernels(swd, name):
    _gives_up(swd, "z_one_row_left", name, (-2,))


def test_stop_option(swd):
    E = _engine(swd, 20, 20, 10, 16, 1)[0]
    assert E.get_option(swd.OPT_RESIDENT_STOP) == 0
    with pytest.raises(swd.SwdError):
        E.set_option(swd.OPT_RESIDENT_STOP, -3)


def test_error_after_a_pass_that_gave_up(swd):
    """A call that returns an error after its on-chip pass gave up leaves nothing behind: the next
    survey, by the step kernels, is stacked."""
    nt = 60
    E, rng, _ = _engine(swd, 100, 100, 10, nt, 6)
    s = swd.ShotSpec(40, 20, np.full(20, 70, np.int32), np.arange(20, 40).astype(np.int32), nt)
    rick, data = swd.ricker_wave(nt, 60.0, 5e-4), rng.standard_normal((20, nt)).astype(np.float32)
    E.set_option(swd.OPT_RESIDENT, 0)
    E.rtm_shot(s, rick, data)
    ref = E.stack(edge_zero=False)
    E.stack_reset()
    E.set_option(swd.OPT_RESIDENT, 1)
    E.set_option(swd.OPT_RESIDENT_STOP, 5)
    with pytest.raises(swd.SwdError):   # angle gathers that were not set up: refused after the forward pass
        E.rtm_shot(s, rick, data, flags=swd.RTM_PREPROCESS | swd.RTM_CIG)
    E.set_option(swd.OPT_RESIDENT_STOP, 0)
    E.set_option(swd.OPT_RESIDENT, 0)
    E.rtm_batch([s], [rick], [data])
    assert np.abs(ref).max() > 0 and np.array_equal(E.stack(edge_zero=False), ref)


RESET = """
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from conftest import load_pkg
swd = load_pkg()
nt = 40
def shot(res):
    E = swd.Engine(100, 60, 10, 4, 5.0, 5.0, 5e-4, nt)
    vp = np.full((128, 88), 2000.0, np.float32)
    E.setup_default(vp, np.full_like(vp, 1000.0))
    E.set_option(swd.OPT_RESIDENT, res)
    s = swd.ShotSpec(40, 20, np.full(9, 50, np.int32), np.arange(15, 24).astype(np.int32), nt)
    out = [E.forward(s, swd.ricker_wave(nt, 60.0, 5e-4)) for _ in range(2)]
    assert E.get_option(swd.OPT_RESIDENT) == res
    E.close()
    return out[1]
ref = shot(0)
assert np.abs(ref).max() > 0 and np.array_equal(shot(1), ref)
assert ctypes.CDLL("libcudart.so.12").cudaDeviceReset() == 0
assert np.array_equal(shot(1), ref)
"""


def test_on_chip_passes_after_a_device_reset(swd):
    """A program that closes its engines, resets its device context and goes on (in a process of its
    own): the on-chip passes keep nothing from before."""
    r = subprocess.run([sys.executable, "-c", RESET, str(ROOT / "tests")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_surveys_keep_their_batches(swd):
    """Surveys of one or two shots go on the chip and leave the batch size untuned; larger ones are tuned
    and batched, also after an on-chip survey and with the on-chip passes switched off between; a last
    shot left over from the batches may go on the chip, and give up there.  The stacks are the same bits."""
    nt = 80
    E, rng, (ntx, ntz) = _engine(swd, 100, 60, 10, nt, 6)
    rick = swd.ricker_wave(nt, 60.0, 5e-4)
    shots = [swd.ShotSpec(30 + 10 * k, 14, np.full(20, 70, np.int32), np.arange(20, 40).astype(np.int32), nt) for k in range(5)]
    data = [rng.standard_normal((20, nt)).astype(np.float32) for _ in shots]

    def stack(n):
        E.stack_reset()
        n0 = E.launch_count()
        E.rtm_batch(shots[:n], [rick] * n, data[:n])
        return E.stack(edge_zero=False), E.launch_count() - n0

    E.set_option(swd.OPT_RESIDENT, 0)
    E.set_option(swd.OPT_BATCH, 1)
    ref = {n: stack(n) for n in (1, 2, 3, 5)}
    E.set_option(swd.OPT_BATCH, 0)
    E.set_option(swd.OPT_RESIDENT, 1)
    for n in (1, 2):
        got = stack(n)
        assert np.array_equal(got[0], ref[n][0]) and got[1] < 0.2 * ref[n][1]
    assert E.get_option(swd.OPT_BATCH_TUNED) == 0
    E.set_option(swd.OPT_RESIDENT, 0)
    assert np.array_equal(stack(5)[0], ref[5][0])
    assert E.get_option(swd.OPT_BATCH_TUNED) == 4   # a batch of four takes about the time of one shot here
    E.set_option(swd.OPT_RESIDENT, 1)
    for n in (3, 5):
        got = stack(n)
        assert np.array_equal(got[0], ref[n][0]) and got[1] < 0.5 * ref[n][1]
    E.set_option(swd.OPT_RESIDENT_STOP, 7)
    assert np.array_equal(stack(5)[0], ref[5][0])
    assert E.get_option(swd.OPT_RESIDENT) == 0
