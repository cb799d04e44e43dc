// resident.cu -- kernels of the on-chip time loops (resident.cuh) and their launcher.
#include <limits.h>
#include <algorithm>
#include "resident.cuh"

namespace swd {

__device__ __forceinline__ ulonglong2 ll_load(const ulonglong2 *p)
{
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void ll_store(ulonglong2 *p, float a, float b, unsigned tag)
{
    unsigned long long u, v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(u) : "r"(__float_as_uint(a)), "r"(tag));
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(__float_as_uint(b)), "r"(tag));
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(u), "l"(v) : "memory");
}
__device__ __forceinline__ bool ll_ok(const ulonglong2 &v, unsigned tag)
{
    return (unsigned)(v.x >> 32) == tag && (unsigned)(v.y >> 32) == tag;
}
__device__ __forceinline__ float2 ll_val(const ulonglong2 &v)
{
    return make_float2(__uint_as_float((unsigned)v.x), __uint_as_float((unsigned)v.y));
}
// four rows of one halo column (or one halo row chunk): two pieces
__device__ __forceinline__ void ll_send4(ulonglong2 *p, float4 v, unsigned tag)
{
    ll_store(p, v.x, v.y, tag);
    ll_store(p + 1, v.z, v.w, tag);
}
// re-reads a piece until it carries the tag; false when it gave up
__device__ __forceinline__ bool ll_wait(const ulonglong2 *p, ulonglong2 &v, unsigned tag)
{
    int n = RES_SPIN;
    while (!ll_ok(v, tag)) {
        if (--n == 0) return false;
        v = ll_load(p);
    }
    return true;
}

// piece offsets inside one (tile, wave, half) area
__device__ __forceinline__ int lx_piece(int side, int j, int row) { return side * 256 + j * 64 + (row >> 1); }
__device__ __forceinline__ int lz_piece(int TX, int side, int col) { return 512 + side * 2 * TX + 2 * col; }

__device__ __forceinline__ float4 mask4(float4 v, unsigned m)
{
    return make_float4(m & 1 ? v.x : 0.f, m & 2 ? v.y : 0.f, m & 4 ? v.z : 0.f, m & 8 ? v.w : 0.f);
}

// NW wavefields, XR columns per warp, at most MW warps, MODE 0 forward / 1 backward (wave 0 source,
// wave 1 receiver) / 2 Born (wave 0 background, wave 1 scattered field) / 3 background with its
// p-update sums S0 written out.  One CTA per SM.
//
// Cells outside an update's guards get a zero coefficient instead of a branch (the field then
// keeps its value), and the CPML terms are formed wherever the warp touches the frame (zero
// profile coefficients elsewhere), so inner and frame warps run the same straight code: every
// tile waits for its neighbours in every half step, so the slowest tile sets the pace.
template <int NW, int XR, int MW, int MODE>
__global__ void __launch_bounds__(32 * MW, 1) k_resident(const ResArgs a)
{
    constexpr int LC = RES_LC, PZ = RES_PZ, TZ = RES_TZ;
    const int TX = a.TX, GX = a.GX, GZ = a.GZ;
    const Geo &g = a.g;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tid = threadIdx.x, nthr = blockDim.x;
    const int bz = blockIdx.x % GZ, bx = blockIdx.x / GZ;
    const int X0 = bx * TX, Z0 = bz * TZ, c0 = warp * XR, z0 = Z0 + 4 * lane;
    const bool hl = bx > 0, hr = bx < GX - 1, ht = bz > 0, hb = bz < GZ - 1;
    const int ntx = g.ntx, ntz = g.ntz, ldz = g.ldz;

    // an earlier pass gave up: do not wait for anyone
    if (*a.err || (a.stop < 0 && blockIdx.x == 0)) return;
    extern __shared__ float4 smem4[];
    float *sm = (float *)smem4;
    const int psz = (TX + 8) * PZ, vsz = (TX + 8) * TZ;
    float *xp = sm + NW * (psz + vsz);          // axh, bxh, ax, bx
    float *zp = xp + 4 * TX;                    // azh, bzh, az, bz
    int *wcs = (int *)(zp + 4 * TZ);            // well of each column
    float *hzs = (float *)(wcs + ((TX + 3) & ~3));   // vz rows above and below the tile: [NW][2][TX][4]
    unsigned *tab = (unsigned *)(hzs + NW * 8 * TX);   // halo pieces to receive: piece << 16 | shared float2
    __shared__ int ntab[2];
    auto P = [&](int k, int c, int row) -> float * { return sm + k * psz + (c + 4) * PZ + 4 + row; };
    auto V = [&](int k, int c, int row) -> float * { return sm + NW * psz + k * vsz + (c + 4) * TZ + row; };
    const bool in = z0 < ntz;
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    auto cell = [&](int i) { return (size_t)(X0 + c0 + i) * ldz + z0; };
    auto has = [&](int i) { return in && X0 + c0 + i < ntx; };

    // ---- state and tables into shared memory and registers
    for (int j = tid; j < NW * (psz + vsz); j += nthr) sm[j] = 0.f;
    for (int j = tid; j < NW * 8 * TX; j += nthr) hzs[j] = 0.f;
    int zframe = 0, xframe = 0;
    for (int j = tid; j < TX; j += nthr) {
        const int x = X0 + j;
        const bool ok = x < ntx;
        xp[j] = ok ? a.c.axh[x] : 0.f;
        xp[TX + j] = ok ? a.c.bxh[x] : 0.f;
        xp[2 * TX + j] = ok ? a.c.ax[x] : 0.f;
        xp[3 * TX + j] = ok ? a.c.bx[x] : 0.f;
        wcs[j] = ok && a.wells.wcol ? a.wells.wcol[x] : -1;
        xframe |= xp[j] != 0.f || xp[2 * TX + j] != 0.f;
    }
    for (int j = tid; j < TZ; j += nthr) {
        const int z = Z0 + j;
        const bool ok = z < ntz;
        zp[j] = ok ? a.c.azh[z] : 0.f;
        zp[TZ + j] = ok ? a.c.bzh[z] : 0.f;
        zp[2 * TZ + j] = ok ? a.c.az[z] : 0.f;
        zp[3 * TZ + j] = ok ? a.c.bz[z] : 0.f;
        zframe |= zp[j] != 0.f || zp[2 * TZ + j] != 0.f;
    }
    if (tid < 2) ntab[tid] = 0;
    zframe = __syncthreads_or(zframe);   // the tile has rows / columns of the CPML frame
    xframe = __syncthreads_or(xframe);
    // ---- receive lists: half 1 (vx columns), then half 0 (p columns and rows)
    const int np = res_pieces(TX), tabcap = NW * (448 + 4 * TX);
    auto HZ = [&](int k, int side, int c) -> float * { return hzs + ((k * 2 + side) * TX + c) * 4; };
    for (int k = 0; k < NW; k++)
        for (int j = tid; j < 512 + 4 * TX; j += nthr) {
            int dp = -1, dv = -1;
            if (j < 512) {
                const int side = j >> 8, col = (j >> 6) & 3, row = (j & 63) * 2;
                if (side ? hr : hl) {
                    if (side || col > 0) dp = (int)(P(k, side ? TX + col : col - 4, row) - sm);
                    if (!side || col < 3) dv = (int)(V(k, side ? TX + col : col - 4, row) - sm);
                }
            } else {
                const int jj = j - 512, side = jj >= 2 * TX, r = jj - side * 2 * TX;
                if (side ? hb : ht) {
                    dp = (int)(P(k, r >> 1, (side ? TZ : -4) + (r & 1) * 2) - sm);
                    dv = (int)(HZ(k, side, r >> 1) + (r & 1) * 2 - sm);
                }
            }
            const unsigned at = (unsigned)(k * 2 * np + j) << 16;   // piece within the tile's area
            if (dp >= 0) tab[tabcap + atomicAdd(&ntab[0], 1)] = at | (unsigned)(dp >> 1);
            if (dv >= 0) tab[atomicAdd(&ntab[1], 1)] = (at + ((unsigned)np << 16)) | (unsigned)(dv >> 1);
        }
    float4 vz[NW][XR];
#pragma unroll
    for (int k = 0; k < NW; k++) {
#pragma unroll
        for (int i = 0; i < XR; i++) {
            vz[k][i] = zero4;
            if (has(i)) {
                st4(P(k, c0 + i, 4 * lane), ld4(a.w[k].p + cell(i)));
                st4(V(k, c0 + i, 4 * lane), ld4(a.w[k].vx + cell(i)));
                vz[k][i] = ld4(a.w[k].vz + cell(i));
            }
        }
        // pressure halo of the first velocity half (the velocity halos arrive by exchange)
        for (int j = warp; j < 8; j += nthr >> 5) {
            const int c = j < 4 ? j - 4 : TX + j - 4, x = X0 + c;
            if (x >= 0 && x < ntx && in) st4(P(k, c, 4 * lane), ld4(a.w[k].p + (size_t)x * ldz + z0));
        }
        for (int c = tid; c < TX; c += nthr) {
            const int x = X0 + c;
            if (x >= ntx) continue;
            if (ht) st4(P(k, c, -4), ld4(a.w[k].p + (size_t)x * ldz + Z0 - 4));
            if (hb) st4(P(k, c, TZ), ld4(a.w[k].p + (size_t)x * ldz + Z0 + TZ));
        }
    }
    // ---- own-cell arrays, one slot of TX columns each, in the order ck, cbx, cbz, then phi_p_x,
    // phi_p_z, phi_v_x, phi_v_z of each CPML wave, then the image sums and kap (backward)
    constexpr int NC = MODE == 1 ? 1 : NW, S_CK = 0, S_CBX = 1, S_CBZ = 2, S_PHI = 3, S_I = S_PHI + 4 * NC, S_S = S_I + 1, S_KAP = S_I + 2;
    constexpr int S_DK = S_I;   // Born
    constexpr bool BORN = MODE == 2, SUMS = MODE >= 2;
    float *slots = hzs + ((NW * 8 * TX + 2 * tabcap + 3) & ~3);
    auto keep = [&](int slot, const float *gp) {
#pragma unroll
        for (int i = 0; i < XR; i++)
            st4(slots + slot * TX * TZ + (c0 + i) * TZ + 4 * lane, has(i) ? ld4(gp + cell(i)) : zero4);
    };
    keep(S_CK, a.m.ck);
    keep(S_CBX, a.m.cbx);
    keep(S_CBZ, a.m.cbz);
#pragma unroll
    for (int k = 0; k < NC; k++) {
        const Wave &w = a.w[MODE == 1 ? 1 : k];
        keep(S_PHI + 4 * k, w.ppx);
        keep(S_PHI + 4 * k + 1, w.ppz);
        keep(S_PHI + 4 * k + 2, w.pvx);
        keep(S_PHI + 4 * k + 3, w.pvz);
    }
    if (MODE == 1) {
        keep(S_I, a.Ip);
        keep(S_S, a.Sp);
        keep(S_KAP, a.m.kap);
    }
    if (BORN) keep(S_DK, a.dkappa);
    __syncthreads();
    const int nV = ntab[1], nP = ntab[0];

    // ---- exchange areas of the four neighbours, at this warp's columns: half 0 p, half 1 velocities
    ulonglong2 *ll = (ulonglong2 *)a.ll;
    const int astep = 2 * np;   // pieces between two waves of a tile
    const int aL = (blockIdx.x - GZ) * NW * astep + lx_piece(1, c0, 4 * lane);
    const int aR = (blockIdx.x + GZ) * NW * astep + lx_piece(0, c0 - (TX - LC), 4 * lane);
    const int aT = ((int)blockIdx.x - 1) * NW * astep + lz_piece(TX, 1, c0);
    const int aB = (blockIdx.x + 1) * NW * astep + lz_piece(TX, 0, c0);
    const bool zsend = (lane == 0 && ht) || (lane == 31 && hb);
    const int aZ = lane == 0 ? aT : aB;
    const bool xsend = (hl && c0 < LC) || (hr && c0 + XR > TX - LC);
    // frame and guard state of the warp (x uniform per column)
    const bool mk = !(X0 + c0 >= g.lx0 && X0 + c0 + XR <= g.lx1 && Z0 >= g.lz0 && Z0 + TZ <= g.lz1);
    const int x0 = X0 + c0;
    bool fx = false;
#pragma unroll
    for (int i = 0; i < XR; i++) fx |= xp[c0 + i] != 0.f || xp[2 * TX + c0 + i] != 0.f;
    const bool fz = zframe != 0;
    unsigned mp = 0, mv = 0, mi = 0, mw = 0;
    int zband = 0, zoff = 0, xmid = 0;   // strip rows of this thread: top or bottom band, middle rows
    const int nx = ntx - 2 * g.pmlc, nzs = ntz - 2 * g.pmlc - 2 * LC;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int z = z0 + q;
        if (z >= LC && z <= ntz - LC) mp |= 1u << q;
        if (z >= LC - 1 && z <= ntz - LC - 1) mv |= 1u << q;
        if (z >= g.pmlc && z <= ntz - g.pmlc - 1) {
            mi |= 1u << q;
            if (z < g.pmlc + LC) { zband |= 1 << q; zoff = z0 - g.pmlc; }
            else if (z >= ntz - g.pmlc - LC) { zband |= 1 << q; zoff = LC * nx + z0 - (ntz - g.pmlc - LC); }
            else xmid |= 1 << q;
        }
        if (z <= ntz - 1) mw |= 1u << q;
    }
    // the strips' offset of (x, z0) where x lies in the left or right band, or -1
    auto xstrip = [&](int x) {
        if (x >= g.pmlc && x < g.pmlc + LC) return 2 * LC * nx + (x - g.pmlc) * nzs + z0 - g.pmlc - LC;
        if (x >= ntx - g.pmlc - LC && x < ntx - g.pmlc) return 2 * LC * nx + LC * nzs + (x - (ntx - g.pmlc - LC)) * nzs + z0 - g.pmlc - LC;
        return INT_MIN;
    };
    const bool sx_here = a.sx >= x0 && a.sx < x0 + XR && a.sz >= z0 && a.sz < z0 + 4;
    // the warp's first well column and its traces
    int wi = -1;
    int4 wtr = make_int4(-1, -1, -1, -1);
#pragma unroll
    for (int i = XR - 1; i >= 0; i--)
        if (wcs[c0 + i] >= 0) wi = i;
    if (wi >= 0 && in) {
        wtr = __ldg(reinterpret_cast<const int4 *>(a.wells.wmap + (size_t)wcs[c0 + wi] * ldz + z0));
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (z0 + q >= ntz) (&wtr.x)[q] = -1;
    }
    auto xin = [&](int x) { return x >= g.pmlc && x <= ntx - g.pmlc - 1; };
    bool bad = false;
    // receives the pieces of a list: up to four a thread in flight at once
    const ulonglong2 *llme = ll + (size_t)blockIdx.x * NW * 2 * np;
    auto receive = [&](const unsigned *t, int n, unsigned tag) {
        for (int j0 = tid; j0 < n; j0 += 4 * nthr) {
            unsigned e[4];
            ulonglong2 v[4];
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const int j = j0 + m * nthr;
                e[m] = j < n ? t[j] : 0xffffffffu;
                if (j < n) v[m] = ll_load(llme + (e[m] >> 16));
            }
#pragma unroll
            for (int m = 0; m < 4; m++)
                if (e[m] != 0xffffffffu) {
                    if (!ll_wait(llme + (e[m] >> 16), v[m], tag)) bad = true;
                    reinterpret_cast<float2 *>(sm)[e[m] & 0xffffu] = ll_val(v[m]);
                }
        }
    };

#pragma unroll 1
    for (int s = 0; s < a.nsteps; s++) {
        const int it = MODE == 1 ? a.t0 - s : a.t0 + s;
        const unsigned tag = a.epoch + 1u + (unsigned)s;
        // the thread's addresses are formed anew in every step (opaque copies), so that the compiler
        // does not keep dozens of loop invariants in registers and spill the fields for them
        int co = c0, lo = lane;
        asm volatile("" : "+r"(co), "+r"(lo));
        float *Pb = sm + (co + 4) * PZ + 4 + 4 * lo, *Vb = sm + NW * psz + (co + 4) * TZ + 4 * lo;
        const float *xpb = xp + co, *zpb = zp + 4 * lo;
        float *Sb = slots + co * TZ + 4 * lo;
        const int ss = TX * TZ;
        auto own = [&](int slot, int i) { return ld4(Sb + slot * ss + i * TZ); };   // own-cell array, column i
        float4 inj = zero4;
        if (MODE == 1 && wi >= 0) {
#pragma unroll
            for (int q = 0; q < 4; q++)
                if ((&wtr.x)[q] >= 0) {
                    const float *rd = a.rdata + (size_t)(&wtr.x)[q] * a.nt + it;
                    el(inj, q) = *rd;
                    if (it >= 32) prefetch_l2(rd - 32);
                }
        }
        // =========================== velocity half ===========================
#pragma unroll
        for (int k = 0; k < NW; k++) {
            const bool src = MODE == 1 && k == 0;            // reconstructed source: interior only, no CPML, -dt
            const bool wide = MODE == 1 && k == 1;           // receiver: wide guards, negated spacing
            const int phi = S_PHI + (MODE == 1 ? 0 : 4 * k);
            const float (&tx)[MAXLC] = wide ? g.ncx : g.cx;
            const float (&tz)[MAXLC] = wide ? g.ncz : g.cz;
            float *Pk = Pb + k * psz, *Vk = Vb + k * vsz;
            if (!(src && it >= a.nt - 2)) {                  // the source starts from the final forward velocities
                const float4 az = ld4(zpb);
                const bool zf = !src && fz && (az.x != 0.f || az.y != 0.f || az.z != 0.f || az.w != 0.f);
                float4 pw[XR + 2 * LC - 1];
#pragma unroll
                for (int j = 0; j < 2 * LC - 1; j++) pw[j] = ld4(Pk + (j - (LC - 1)) * PZ);
#pragma unroll
                for (int i = 0; i < XR; i++) {
                    const int x = x0 + i;
                    float4 cX = own(S_CBX, i), cZ = own(S_CBZ, i);
                    float4 ff = zero4, fg = zero4;
                    const float ax = !src && fx ? xpb[i] : 0.f;
                    if (!src && fx && ax != 0.f) ff = own(phi, i);
                    if (zf) fg = own(phi + 1, i);
                    float4 v = ld4(Vk + i * TZ);
                    pw[i + 2 * LC - 1] = ld4(Pk + (i + LC) * PZ);
                    const float4 up = ld4(Pk + i * PZ - 4), dn = ld4(Pk + i * PZ + 4), ow = pw[i + LC - 1];
                    float4 d = zero4, e = zero4;
#pragma unroll
                    for (int ic = 0; ic < LC; ic++)
#pragma unroll
                        for (int q = 0; q < 4; q++) el(d, q) += tx[ic] * (elc(pw[i + LC + ic], q) - elc(pw[i + LC - 1 - ic], q));
                    const float w[12] = {up.x, up.y, up.z, up.w, ow.x, ow.y, ow.z, ow.w, dn.x, dn.y, dn.z, dn.w};
#pragma unroll
                    for (int q = 0; q < 4; q++)
#pragma unroll
                        for (int ic = 0; ic < LC; ic++) el(e, q) += tz[ic] * (w[4 + q + ic + 1] - w[4 + q - ic]);
                    if (!src && fx && ax != 0.f) {
                        const float bxv = xpb[TX + i];
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            el(ff, q) = bxv * elc(ff, q) + ax * elc(d, q);
                            el(d, q) = elc(d, q) + elc(ff, q);
                        }
                        st4(Sb + (phi) * ss + i * TZ, ff);
                    }
                    if (zf) {
                        const float4 bzv = ld4(zpb + TZ);
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            el(fg, q) = elc(az, q) != 0.f ? elc(bzv, q) * elc(fg, q) + elc(az, q) * elc(e, q) : 0.f;
                            el(e, q) = elc(e, q) + elc(fg, q);
                        }
                        st4(Sb + (phi + 1) * ss + i * TZ, fg);
                    }
                    if (mk) {
                        cX = mask4(cX, src ? (xin(x) ? mi : 0u) : (x >= LC - 1 && x <= ntx - LC - 1) ? (wide ? mw : mp) : 0u);
                        cZ = mask4(cZ, src ? (xin(x) ? mi : 0u) : (wide ? x < ntx : (x >= LC && x <= ntx - LC)) ? mv : 0u);
                    }
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        el(v, q) = (src ? -elc(cX, q) : elc(cX, q)) * elc(d, q) + elc(v, q);
                        el(vz[k][i], q) = (src ? -elc(cZ, q) : elc(cZ, q)) * elc(e, q) + elc(vz[k][i], q);
                    }
                    st4(Vk + i * TZ, v);
                }
            }
            if (xsend) {
#pragma unroll
                for (int i = 0; i < XR; i++) {
                    const int c = co + i;
                    if (hl && c < LC - 1) ll_send4(ll + aL + k * astep + np + 64 * i, ld4(Vk + i * TZ), tag);
                    if (hr && c >= TX - LC) ll_send4(ll + aR + k * astep + np + 64 * i, ld4(Vk + i * TZ), tag);
                }
            }
            if (zsend) {
#pragma unroll
                for (int i = 0; i < XR; i++) ll_send4(ll + aZ + k * astep + np + 2 * i, vz[k][i], tag);
            }
        }
        receive(tab, nV, tag);
        if (__syncthreads_or(bad)) break;

        // =========================== pressure half ===========================
        asm volatile("" : "+r"(co), "+r"(lo));
        Pb = sm + (co + 4) * PZ + 4 + 4 * lo;
        Vb = sm + NW * psz + (co + 4) * TZ + 4 * lo;
        xpb = xp + co;
        zpb = zp + 4 * lo;
        Sb = slots + co * TZ + 4 * lo;
        float4 dp[MODE == 0 ? 1 : XR];   // backward: the source's p-update sum of interior cells; Born: field 0's of updated cells
#pragma unroll
        for (int k = 0; k < NW; k++) {
            const bool src = MODE == 1 && k == 0;
            const bool rcv = MODE == 1 && k == 1;
            const int phi = S_PHI + (MODE == 1 ? 0 : 4 * k);
            const float (&tx)[MAXLC] = rcv ? g.ncx : g.cx;
            const float (&tz)[MAXLC] = rcv ? g.ncz : g.cz;
            float *Pk = Pb + k * psz, *Vk = Vb + k * vsz;
            const float *hzk = hzs + (k * 2 * TX + co) * 4 + (lo == 31 ? 4 * TX : 0);   // row neighbours of lanes 0 and 31
            const float4 az = ld4(zpb + 2 * TZ);
            const bool zf = !src && fz && (az.x != 0.f || az.y != 0.f || az.z != 0.f || az.w != 0.f);
            float4 vw[XR + 2 * LC - 1];
#pragma unroll
            for (int j = 0; j < 2 * LC - 1; j++) vw[j] = ld4(Vk + (j - LC) * TZ);
#pragma unroll
            for (int i = 0; i < XR; i++) {
                const int x = x0 + i;
                float4 kc = own(S_CK, i), ff = zero4, f = zero4;
                const float ax = !src && fx ? xpb[2 * TX + i] : 0.f;
                if (!src && fx && ax != 0.f) ff = own(phi + 2, i);
                if (zf) f = own(phi + 3, i);
                vw[i + 2 * LC - 1] = ld4(Vk + (i + LC - 1) * TZ);
                float4 p = ld4(Pk + i * PZ);
                // z window of vz: rows -4 .. 6 around the four
                const float4 o = vz[k][i], hz = ld4(hzk + 4 * i);
                float4 up, dn;
                up.x = __shfl_up_sync(0xffffffffu, o.x, 1);
                up.y = __shfl_up_sync(0xffffffffu, o.y, 1);
                up.z = __shfl_up_sync(0xffffffffu, o.z, 1);
                up.w = __shfl_up_sync(0xffffffffu, o.w, 1);
                dn.x = __shfl_down_sync(0xffffffffu, o.x, 1);
                dn.y = __shfl_down_sync(0xffffffffu, o.y, 1);
                dn.z = __shfl_down_sync(0xffffffffu, o.z, 1);
                if (lo == 0) up = hz;
                if (lo == 31) dn = hz;
                const float w[11] = {up.x, up.y, up.z, up.w, o.x, o.y, o.z, o.w, dn.x, dn.y, dn.z};
                float4 d = zero4, e = zero4;
#pragma unroll
                for (int ic = 0; ic < LC; ic++)
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        el(d, q) += tx[ic] * (elc(vw[i + LC + ic], q) - elc(vw[i + LC - 1 - ic], q));
                        el(e, q) += tz[ic] * (w[4 + q + ic] - w[4 + q - ic - 1]);
                    }
                const unsigned im = mk ? (xin(x) ? mi : 0u) : 15u;
                if (src) {
#pragma unroll
                    for (int q = 0; q < 4; q++) el(d, q) = elc(d, q) + elc(e, q);
                    if (mk) d = mask4(d, im);
                    dp[i] = d;
#pragma unroll
                    for (int q = 0; q < 4; q++) el(p, q) = (-elc(kc, q)) * elc(d, q) + elc(p, q);
                    if (sx_here && x == a.sx) {
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (a.sz == z0 + q) el(p, q) -= a.wav0[it + 1];
                    }
                } else {
                    if (fx && ax != 0.f) {
                        const float bxv = xpb[3 * TX + i];
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            el(ff, q) = bxv * elc(ff, q) + ax * elc(d, q);
                            el(d, q) = elc(d, q) + elc(ff, q);
                        }
                        st4(Sb + (phi + 2) * ss + i * TZ, ff);
                    }
                    if (zf) {
                        const float4 bzv = ld4(zpb + 3 * TZ);
#pragma unroll
                        for (int q = 0; q < 4; q++) el(f, q) = elc(az, q) != 0.f ? elc(bzv, q) * elc(f, q) + elc(az, q) * elc(e, q) : 0.f;
                        st4(Sb + (phi + 3) * ss + i * TZ, f);
                    }
                    const unsigned gp = mk ? ((x >= LC && x <= ntx - LC) ? mp : 0u) : 15u;
                    if (mk) kc = mask4(kc, gp);
                    if (SUMS && k == 0) {
#pragma unroll
                        for (int q = 0; q < 4; q++) el(dp[i], q) = elc(d, q) + elc(e, q) + elc(f, q);
                        if (mk) dp[i] = mask4(dp[i], gp);
                        if (MODE == 3 && has(i)) st4(a.s0 + (size_t)(it % a.s0_mod) * a.s0_stride + cell(i), dp[i]);
                    }
#pragma unroll
                    for (int q = 0; q < 4; q++) el(p, q) = elc(kc, q) * (elc(d, q) + elc(e, q) + elc(f, q)) + elc(p, q);
                    if (BORN && k == 1) {   // secondary source of the scattered field
                        const float4 dk = own(S_DK, i);
#pragma unroll
                        for (int q = 0; q < 4; q++) el(p, q) += g.dt * elc(dk, q) * elc(dp[i], q);
                    }
                    if (MODE != 1 && sx_here && x == a.sx) {
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (a.sz == z0 + q) el(p, q) += (k == 0 ? a.wav0[it] : a.wav1[it]);
                    }
                    if (rcv && wi >= 0) {   // hard injection of the data
                        if (i == wi) {
#pragma unroll
                            for (int q = 0; q < 4; q++)
                                if ((&wtr.x)[q] >= 0) el(p, q) = elc(inj, q);
                        } else if (wcs[co + i] >= 0 && in) {
                            const int4 tr = __ldg(reinterpret_cast<const int4 *>(a.wells.wmap + (size_t)wcs[co + i] * ldz + z0));
                            const int t[4] = {tr.x, tr.y, tr.z, tr.w};
#pragma unroll
                            for (int q = 0; q < 4; q++)
                                if (t[q] >= 0 && z0 + q < ntz) el(p, q) = a.rdata[(size_t)t[q] * a.nt + it];
                        }
                    }
                }
                st4(Pk + i * PZ, p);
                if (rcv) {   // imaging condition, FP32 block sums folded into FP64 (image4)
                    float4 pi = own(S_I, i), ps = own(S_S, i);
                    const float4 kp = own(S_KAP, i);
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const float dq = elc(kp, q) * elc(dp[i], q);
                        el(pi, q) = fmaf(dq, elc(p, q), elc(pi, q));
                        el(ps, q) = fmaf(dq, dq, elc(ps, q));
                    }
                    if (it % IMG_BLOCK == 0) {
                        double *I = a.I + cell(i), *S = a.S + cell(i);
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (im >> q & 1) {
                                I[q] += (double)elc(pi, q);
                                S[q] += (double)elc(ps, q);
                            }
                        pi = zero4;
                        ps = zero4;
                    }
                    st4(Sb + (S_I) * ss + i * TZ, pi);
                    st4(Sb + (S_S) * ss + i * TZ, ps);
                }
            }
            if (src && mk && mi) {   // boundary strips over the reconstructed pressure
                const float *sp = (const float *)a.strips.buf + (size_t)it * a.strips.slen;
                const size_t ahead = 8 * (size_t)a.strips.slen;
#pragma unroll
                for (int i = 0; i < XR; i++) {
                    const int x = x0 + i;
                    if (!xin(x)) continue;
                    float *pc = Pk + i * PZ;
                    if (zband) {
                        const float *t = sp + zoff + (x - g.pmlc) * LC;
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (zband >> q & 1) {
                                pc[q] = t[q];
                                if (it >= 8) prefetch_l2(t + q - ahead);
                            }
                    }
                    const int xo = xstrip(x);
                    if (xo != INT_MIN) {
                        const float *t = sp + xo;
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (xmid >> q & 1) pc[q] = t[q];
                        if ((xmid & 1) && it >= 8) prefetch_l2(t - ahead);
                    }
                }
            }
            // ---- seams
            if (xsend) {
#pragma unroll
                for (int i = 0; i < XR; i++) {
                    const int c = co + i;
                    if (hl && c < LC) ll_send4(ll + aL + k * astep + 64 * i, ld4(Pk + i * PZ), tag);
                    if (hr && c >= TX - (LC - 1)) ll_send4(ll + aR + k * astep + 64 * i, ld4(Pk + i * PZ), tag);
                }
            }
            if (zsend) {
#pragma unroll
                for (int i = 0; i < XR; i++) ll_send4(ll + aZ + k * astep + 2 * i, ld4(Pk + i * PZ), tag);
            }
        }
        if (MODE != 1) {   // records (Born: of the scattered field) and strips, nobody waits for them
            if (wi >= 0 && in) {
#pragma unroll
                for (int i = 0; i < XR; i++) {
                    const int wc = wcs[co + i];
                    if (wc < 0 || !a.seis) continue;
                    const float4 p = ld4(Pb + (BORN ? psz : 0) + i * PZ);
                    int4 tr = wtr;
                    if (i != wi) tr = __ldg(reinterpret_cast<const int4 *>(a.wells.wmap + (size_t)wc * ldz + z0));
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if ((&tr.x)[q] >= 0 && z0 + q < ntz) a.seis[(size_t)(&tr.x)[q] * a.nt + it] = elc(p, q);
                    if (a.colmap) {
                        const float4 h = ld4(Pb + (NW - 1) * psz + i * PZ);
                        float4 *cb = reinterpret_cast<float4 *>(a.colbuf + ((size_t)wc * a.nt + it) * ldz + z0);
                        cb[0] = make_float4(p.x, h.x, p.y, h.y);
                        cb[1] = make_float4(p.z, h.z, p.w, h.w);
                    }
                }
            }
            if (a.strips.buf && mk && mi) {
                float *sp = (float *)a.strips.buf + (size_t)it * a.strips.slen;
#pragma unroll
                for (int i = 0; i < XR; i++) {
                    const int x = x0 + i;
                    if (!xin(x)) continue;
                    const float4 p = ld4(Pb + i * PZ);
                    if (zband) {
                        float *t = sp + zoff + (x - g.pmlc) * LC;
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (zband >> q & 1) t[q] = elc(p, q);
                    }
                    const int xo = xstrip(x);
                    if (xo != INT_MIN) {
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (xmid >> q & 1) sp[xo + q] = elc(p, q);
                    }
                }
            }
        }
        // pressure halos for the next velocity half
        if (s + 1 < a.nsteps) receive(tab + tabcap, nP, tag);
        if (__syncthreads_or(bad)) break;
    }
    if (__syncthreads_or(bad || (a.stop > 0 && blockIdx.x == 0))) {
        if (tid == 0) { *a.err = 1; *(volatile int *)a.host_err = 1; }
        return;
    }
    // ---- final state.  None after a backward pass: nobody reads it, and where a tile gave up in one of
    // the last steps the pass runs again from the forward pass's final fields, which the tiles that got
    // through must not have overwritten.
#pragma unroll
    for (int k = 0; k < (MODE == 1 ? 0 : NW); k++)
#pragma unroll
        for (int i = 0; i < XR; i++)
            if (has(i)) {
                st4(a.w[k].p + cell(i), ld4(P(k, c0 + i, 4 * lane)));
                st4(a.w[k].vx + cell(i), ld4(V(k, c0 + i, 4 * lane)));
                st4(a.w[k].vz + cell(i), vz[k][i]);
                if (SUMS) {   // a piece of a pass: the CPML memories go on in the next one
                    const float *q = slots + (S_PHI + 4 * k) * TX * TZ + (c0 + i) * TZ + 4 * lane;
                    st4(a.w[k].ppx + cell(i), ld4(q));
                    st4(a.w[k].ppz + cell(i), ld4(q + TX * TZ));
                    st4(a.w[k].pvx + cell(i), ld4(q + 2 * TX * TZ));
                    st4(a.w[k].pvz + cell(i), ld4(q + 3 * TX * TZ));
                }
            }
}

bool res_plan(int ntx, int ntz, int pmlc, int nsm, size_t smem_max, int nw, bool born, ResPlan *p)
{
    if (ntx < 48 || ntz < 48 || !strip_bands_apart(ntz, pmlc, RES_LC)) return false;
    p->nw = nw;
    p->GZ = (ntz + RES_TZ - 1) / RES_TZ;
    const int gx = nsm / p->GZ;
    if (gx < 1) return false;
    const int need = std::max((ntx + gx - 1) / gx, 2 * RES_LC);   // halos come from direct neighbours only
    p->XR = need <= RES_MAXW1 ? 1 : 2;
    p->nwarps = (need + p->XR - 1) / p->XR;
    if (p->XR == 2 && p->nwarps > RES_MAXW2) return false;
    p->TX = p->XR * p->nwarps;
    p->GX = (ntx + p->TX - 1) / p->TX;
    p->smem = res_smem(p->TX, nw) + (born ? sizeof(float) * p->TX * RES_TZ : 0);
    p->ll_bytes = sizeof(ulonglong2) * (size_t)p->GX * p->GZ * nw * 2 * res_pieces(p->TX);
    return p->smem + 1024 <= smem_max;   // 1 KB: static shared memory
}

template <int NW, int XR, int MW, int MODE>
static cudaError_t launch_res(const ResArgs &a, const ResPlan &p, cudaStream_t st)
{
    const void *fn = (const void *)k_resident<NW, XR, MW, MODE>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem);
    if (e != cudaSuccess) return e;
    void *args[1] = {(void *)&a};
    return cudaLaunchCooperativeKernel(fn, dim3(p.GX * p.GZ), dim3(32 * p.nwarps), args, p.smem, st);
}

template <int NW, int MODE>
static cudaError_t launch_xr(const ResArgs &a, const ResPlan &p, cudaStream_t st)
{
    if (p.XR == 2) return launch_res<NW, 2, RES_MAXW2, MODE>(a, p, st);
    return p.nwarps <= RES_MAXW2 ? launch_res<NW, 1, RES_MAXW2, MODE>(a, p, st) : launch_res<NW, 1, RES_MAXW1, MODE>(a, p, st);
}

cudaError_t res_launch(const ResArgs &a, const ResPlan &p, int mode, cudaStream_t st)
{
    if (mode == 1) return launch_xr<2, 1>(a, p, st);
    if (mode == 2) return launch_xr<2, 2>(a, p, st);
    if (mode == 3) return launch_xr<1, 3>(a, p, st);
    return p.nw == 2 ? launch_xr<2, 0>(a, p, st) : launch_xr<1, 0>(a, p, st);
}

}  // namespace swd
