// resident.cuh -- time loops whose wavefields stay on the chip between steps (sm_100a).
//
// One cooperative launch runs a whole pass.  The grid is cut into tiles of TX columns x 128 rows,
// one CTA per tile, at most one per SM.  A CTA keeps its tile's fields from the first step to the
// last: p, vx, the CPML memories, the coefficients and the image sums in shared memory, vz in
// registers (only a cell's own thread and its two neighbour lanes read it).  A step then moves no
// grid array at all; what is left of it is the exchange between tiles and the latency of one
// column's arithmetic, and the two launches per step become two block barriers.
//
// What bounds it: latency.  On 401 x 201 (141 tiles) a forward step takes about 7,000 cycles: two
// waits of 1,650-2,100 for the neighbours' words (a store and a load through L2 each), 1,300 for
// the velocity half and 2,000 for the pressure half of one column per warp.
//
// Measured per time step (B200, 30-cell frame): RTM, forward plus backward, 401 x 201 18.2 -> 9.7
// us, 801 x 401 20.0 -> 14.1 us, 100 x 60 17.0 -> 8.4 us; modelling with the Hilbert twin
// 401 x 201 10.3 -> 5.3 us, 801 x 401 11.1 -> 7.8 us; Born modelling with checkpoints every 64 steps
// 401 x 201 10.3 -> 5.5 us, 801 x 401 10.8 -> 8.0 us.
//
// A warp owns XR adjacent columns of the tile, a lane four rows of them, as in the plain kernels;
// the x taps come from a register window over the neighbouring columns.  One column per warp up to
// 12 columns (168 registers a thread; 100 x 60: 8.4 us per RTM step, with 128 registers 9.1), up to
// 16 still one (128 registers; 600 x 300: 10.8 us, two columns per warp 13.2), then two up to 24:
// with more columns a thread's window and vz no longer fit in registers, and the spills cost more
// than the launches (1601 x 801 with 7 columns per warp: 65 us per RTM step, the step kernels 39).
//
// Neighbouring tiles exchange what the stencil reads across the seam (LC columns of vx, LC rows
// of vz after the velocity half; LC columns and rows of p after the pressure half) through
// global memory as 8-byte words {value, tag}.  A word is written and read by one 64-bit access,
// so a word that carries the expected tag carries its value: no fence and no separate flag.  The
// tag grows by one each step and from launch to launch.  One slot per word is enough: a tile
// writes a word again only after it has received the neighbour's later words of the other half
// step, which the neighbour sends after it has read this one.  Every wait gives up after
// RES_SPIN tries, sets the error word and ends the kernel; the host then runs the pass with the
// plain kernels.
//
// The per-cell arithmetic is the plain kernels' (prop.cuh), tap by tap in the same order, so the
// results are the same bits.
#pragma once
#include "prop.cuh"
#include "rules.h"

namespace swd {

constexpr int RES_LC = 4;            // the stencil half length these kernels are built for
constexpr int RES_TZ = 128;          // rows of a tile (32 lanes x 4)
constexpr int RES_PZ = RES_TZ + 8;   // pressure column in shared memory with its halo rows
constexpr int RES_MAXW1 = 16;        // warps of a CTA at most, one column per warp
constexpr int RES_MAXW2 = 12;        // two columns per warp; one column with the larger register budget
constexpr int RES_SPIN = 1 << 22;    // tries of a wait, 0.36 us each
// Steps of a piece at least: Born passes stop at every checkpoint, and a launch that loads and
// stores the whole state costs about 15 to 25 us.  Born plus adjoint pass per step with checkpoints
// every 4 / 8 / 64 steps: 401 x 201 31.2 -> 27.1 / 27.8 -> 21.8 / 24.9 -> 17.4 us, 801 x 401
// 32.5 -> 33.5 / 28.9 -> 27.3 / 26.2 -> 22.2 us.
constexpr int RES_PIECE = 8;

// Tiling of a grid: CTAs GX x GZ, TX = XR * nwarps columns per tile.
struct ResPlan {
    int XR, nwarps, TX, GX, GZ, nw;   // nw: wavefields
    size_t smem, ll_bytes;
};

struct ResArgs {
    Geo g;
    Cpml c;
    Mat m;
    Wave w[2];             // forward: field and Hilbert twin; backward: source and receiver
    const float *wav0, *wav1;
    int sx, sz, nt;
    Wells wells;
    float *seis;           // forward: [r_n][nt] or nullptr
    const int *colmap;     // forward: kz columns wanted when not null
    float2 *colbuf;
    Strips strips;         // FP32 strips: saved (forward) or restored (backward); buf may be nullptr
    const float *rdata;    // backward: injected data
    double *I, *S;
    float *Ip, *Sp;
    const float *dkappa;   // Born: bulk-modulus perturbation
    float *s0;             // p-update sums, slot it % s0_mod
    long long s0_stride;
    int s0_mod;
    int t0, nsteps;        // steps t0, t0 + 1, ... (forward) or t0, t0 - 1, ... (backward)
    int TX, GX, GZ;
    uint4 *ll;             // exchange words
    unsigned epoch;        // tag of the step before the first
    // tests of the recovery: 1 the first tile reports at the end that it gave up, -1 it does not start
    // and its neighbours wait for it in vain; 0: neither
    int stop;
    int *err, *host_err;   // set when a wait gave up; *err also keeps later launches from starting
};

// 16-byte pieces of the exchange area of one (tile, wave, half): 4 left and 4 right columns of
// 128 rows, 4 top and 4 bottom rows of TX columns, two words per piece
__host__ __device__ constexpr int res_pieces(int TX) { return 2 * (4 * RES_TZ) / 2 + 2 * (4 * TX) / 2; }

// shared memory of a tile in bytes: p and vx with their halos, the x profiles (4 TX), the z
// profiles (4 x 128), the well of each column, the vz halo rows and the receive lists, and the
// own-cell arrays (three coefficients and four CPML memories per wave; the backward pass has one
// wave with CPML, kap and two image sums)
__host__ __device__ inline size_t res_smem(int TX, int nw)
{
    return sizeof(float) * ((size_t)nw * (TX + 8) * (RES_PZ + RES_TZ) + 4 * TX + 4 * RES_TZ + ((TX + 3) & ~3) +
                            (size_t)nw * (8 * TX + 2 * (448 + 4 * TX)) + (size_t)(nw == 1 ? 7 : 11) * TX * RES_TZ);
}

// launches nsteps steps; mode 0 forward, 1 backward (plan.nw == 2), 2 Born (plan.nw == 2), 3 forward
// with S0 (plan.nw == 1); modes 2 and 3 may run a pass in pieces
cudaError_t res_launch(const ResArgs &a, const ResPlan &p, int mode, cudaStream_t st);
// tiling of an ntx x ntz grid (pmlc frame cells) on nsm SMs with smem_max bytes of shared memory per
// CTA; false when the wavefields do not fit; born: with the perturbation of mode 2
bool res_plan(int ntx, int ntz, int pmlc, int nsm, size_t smem_max, int nw, bool born, ResPlan *p);

}  // namespace swd
