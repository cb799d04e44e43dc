// rules.h -- sizes for which the engine takes one kernel path or another: plain host functions of
// numbers, without CUDA, so that they can be checked over whole ranges of sizes on the CPU.
#pragma once
#include <cstddef>

namespace swd {

// The on-chip loops and the marches keep one strip offset per thread for its four rows (the rows
// 4k .. 4k + 3 of the padded grid), so no four rows may hold cells of the top strip and of the bottom
// strip.  The strips are Lc rows each at both ends of the ntz - 2 pmlc interior rows; from 2 Lc + 3
// interior rows on, three rows or more lie between them.
inline bool strip_bands_apart(int ntz, int pmlc, int Lc) { return ntz - 2 * pmlc >= 2 * Lc + 3; }

// A march forms its cell index, column times row pitch plus row, in 32 bits (a lane's address is then
// one multiply-add per array).  Grids beyond that keep the step kernels: two copies of the field and
// six more arrays of 2^31 cells leave no room on a device of 180 GB for anything else.
inline bool march_index_fits(int ntx, int ldz) { return (long long)ntx * ldz <= 0x7fffffffLL; }

// Whether a march pays on a grid of so many cells: the tasks that touch the frame (17 columns and 7 more
// to fill the windows, 128 rows of which 112 are their own) may work on no more cells than the grid
// has.  Flat or narrow grids and wide frames have more of them, at twice the instructions each.  Forward
// step with 16-bit strips, us, march / step kernels, with that work as a share of the grid: 4001 x 1601
// 0.26 54.2 / 62.8, 2300 x 2300 with a 200-cell frame 0.56 65.1 / 67.2, 12000 x 500 0.97 74.0 / 72.0,
// 16000 x 400 1.17 92.1 / 81.4, 20000 x 300 1.48 106.2 / 84.1, 40000 x 160 2.38 184.7 / 125.1.
inline bool march_pays(size_t frame_tasks, long long cells) { return (long long)frame_tasks * (17 + 7) * 128 <= cells; }

// Whether operands prefetched into L2 AHEAD_COLS columns ahead are still there when they are read: what a
// pass of so many arrays touches in those columns is at most a quarter of the L2.  RTM backward step,
// us, without / with: 20000 rows 128.8 / 137.0, 15000 rows 126.0 / 127.5, 9000 rows 126.3 / 120.6; forward
// step (6 arrays) 60000 rows 100.4 / 112.5, 30000 rows 78.4 / 73.8; scattered field (10 arrays a launch)
// 30000 rows 152.0 / 175.2, 20000 rows and 3000 columns 1016 / 976, 10000 rows 125.2 / 115.0.
constexpr int AHEAD_COLS = 40;
inline bool ahead_fits(int ldz, int arrays, size_t l2_bytes) { return (size_t)AHEAD_COLS * ldz * sizeof(float) * arrays <= l2_bytes / 4; }

// Whether a smoothing window of this half width works on a tile of doubles in shared memory, on a grid
// of so many blocks (32 x 8 cells).  Wider windows leave an SM fewer blocks and so too few warps for the
// additions' latency, first where the grid is one wave or little more.  Call with the tile / taps from
// memory, us, at half widths 24 / 28 / 32 / 40 / 48: 1669 x 869 (5,500 blocks) 1628 / 2272 / 2984 / 5656 /
// 8881 and 1729 / 2311 / 2978 / 4570 / 6500; 600 x 400 (860 blocks) 312 / 616 / 655 / 1028 / 1506 and
// 344 / 449 / 566 / 861 / 1221.
constexpr int SMOOTH_TILE_WINDOW = 32;
inline bool smooth_tile(int window, long long blocks) { return window <= 24 || (window <= SMOOTH_TILE_WINDOW && blocks >= 4000); }
inline size_t smooth_smem(int w) { return sizeof(double) * (8 + 2 * (size_t)w) * (32 + 2 * (size_t)w); }

}  // namespace swd
