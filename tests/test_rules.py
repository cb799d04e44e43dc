"""The size rules that choose a kernel path (csrc/rules.h), over whole ranges of sizes on the CPU."""
import ctypes as C
import subprocess

import pytest

from conftest import PKG_DIR

WRAP = """
#include "rules.h"
extern "C" {
int bands_apart(int ntz, int pmlc, int Lc) { return swd::strip_bands_apart(ntz, pmlc, Lc); }
int ahead_fits(int ldz, int arrays, size_t l2) { return swd::ahead_fits(ldz, arrays, l2); }
int march_pays(size_t frame_tasks, long long cells) { return swd::march_pays(frame_tasks, cells); }
int smooth_tile(int window, long long blocks) { return swd::smooth_tile(window, blocks); }
long long smooth_smem(int window) { return swd::smooth_smem(window); }
int index_fits(int ntx, int ldz) { return swd::march_index_fits(ntx, ldz); }
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "wrap.cpp").write_text(WRAP)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", f"-I{PKG_DIR / 'csrc'}",
                    "-o", str(d / "rules.so"), str(d / "wrap.cpp")], check=True)
    return C.CDLL(str(d / "rules.so"))


def test_strip_rows_of_a_thread(rules):
    """Wherever the rule lets a grid through, the strip slot a thread forms from its single offset is
    the cell's own slot, and no grid of 11 or more interior rows is turned away."""
    Lc, nx, ix = 4, 20, 7
    wrong = set()
    for nz in range(9, 16):
        for pml in range(1, 45):
            p = pml + Lc
            ntz = nz + 2 * p
            ok = True
            for z0 in range(0, ntz, 4):
                off, own = 0, {}
                for z in range(z0, min(z0 + 4, ntz)):
                    if p <= z < p + Lc:                          # top strip: Lc values per column
                        off, own[z] = z0 - p, z - p
                    elif ntz - p - Lc <= z < ntz - p:            # bottom strip, after the top one
                        off, own[z] = Lc * nx + z0 - (ntz - p - Lc), Lc * nx + z - (ntz - p - Lc)
                ok &= all(off + ix * Lc + z - z0 == s + ix * Lc for z, s in own.items())
            if not ok:
                wrong.add(nz)
            assert rules.bands_apart(ntz, p, Lc) == (nz >= 11)
            assert ok or nz < 11, (nz, pml)
    assert wrong == {9, 10}   # the check does see the grids that must be turned away


def test_march_index_range(rules):
    """Every index a march forms (col * ldz + row, row from -8 to ldz - 4) fits in 32 bits where the
    rule lets the grid through; the largest grid that fits is let through."""
    for ldz in (64, 1696, 46336, 46368, 65536, 1 << 20):
        for ntx in (100, 4069, (2 ** 31 - 1) // ldz, (2 ** 31 - 1) // ldz + 1, 46341, 2 ** 31 // ldz + 100):
            fits = (ntx - 1) * ldz + ldz - 4 < 2 ** 31 and ntx * ldz < 2 ** 31
            assert bool(rules.index_fits(ntx, ldz)) == fits, (ntx, ldz)


def test_smoothing_tiles_leave_room_for_warps(rules):
    """Wherever a tile is used an SM holds at least four blocks of it (227 KB, 1 KB each reserved), six on
    grids of few blocks; the reference's window always uses it."""
    rules.smooth_tile.argtypes, rules.smooth_smem.restype = [C.c_int, C.c_longlong], C.c_longlong
    assert rules.smooth_tile(5, 1)
    for blocks in (1, 500, 3999, 4000, 10 ** 9):
        for w in range(65):
            per_sm = 227 * 1024 // (rules.smooth_smem(w) + 1024)
            if rules.smooth_tile(w, blocks):
                assert per_sm >= (4 if blocks >= 4000 else 6), (w, blocks)


def test_march_wants_little_frame(rules):
    """Frame tasks counted as the launch cuts them (row tiles of 112, frame chunks of 17 columns, lean
    chunks of 33 or more): squarish grids march, flat and narrow ones keep the step kernels."""
    rules.march_pays.argtypes = [C.c_size_t, C.c_longlong]

    def pays(nx, nz, pml, wide):
        p = pml + 4
        ntx, ntz = nx + 2 * p, nz + 2 * p
        frame = 0
        for bz in range(-(-ntz // 112)):
            x, zl = 0, bz * 112 - 8 >= p + 4 and bz * 112 + 120 <= ntz - p - 4
            while x < ntx:
                lean = zl and x - 8 >= p + 4 and x + wide + 8 <= ntx - p - 4
                frame += not lean
                x += wide if lean else 17
        return bool(rules.march_pays(frame, ntx * ntz))

    for grid in ((4001, 1601, 30, 57), (3001, 1403, 30, 33), (2400, 2400, 100, 49), (12000, 500, 30, 33), (400, 15000, 30, 49)):
        assert pays(*grid), grid
    for grid in ((16000, 400, 30, 33), (30000, 200, 10, 33), (60000, 100, 10, 33), (60, 90000, 10, 33)):
        assert not pays(*grid), grid


def test_reads_ahead_stay_in_l2(rules):
    """126 MB of L2: grids of the usual depth read ahead in every pass, tall ones only with few arrays."""
    rules.ahead_fits.argtypes = [C.c_int, C.c_int, C.c_size_t]
    fits = lambda ldz, arrays: bool(rules.ahead_fits(ldz, arrays, 132644864))
    assert fits(1696, 12) and fits(4096, 12) and fits(30080, 6)
    assert not fits(20096, 12) and fits(20096, 10) and not fits(30080, 10) and not fits(60096, 6)
    assert not rules.ahead_fits(64, 6, 0)   # an L2 of unknown size
