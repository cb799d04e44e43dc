// rules.h -- sizes for which the engine takes one kernel path or another: plain host functions of
// numbers, without CUDA, so that they can be checked over whole ranges of sizes on the CPU.
#pragma once

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

}  // namespace swd
