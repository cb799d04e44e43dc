// march.cuh -- forward steps of large grids, velocity and pressure in one launch (sm_100a).
//
// The two launches of a step read and write the fields of a grid that does not fit in L2 twice:
// 48 bytes per cell and wavefield where one pass needs 36 (p, vx, vz in and out, three
// coefficients).  Here one warp makes both halves in one sweep.  A warp holds 128 rows (four per
// lane) and marches along x over C columns; at column j it has the new vx of j, and with it
// everything the pressure of column j - 3 needs:
//   vx(j)      from p(j-3 .. j+4), a window of eight columns in registers,
//   vz(j-3)    from p(j-3), rows of the neighbour lanes by shuffles,
//   p(j-3)     from the last eight new vx columns and the new vz.
// Nothing is shared between warps: the 16 outer rows of a warp (of which 112 are its own) and the
// seven columns ahead of its first are computed twice, from the same inputs, so every field is
// double-buffered (a step reads one copy and writes the other).  Each array's column is copied by
// cp.async into a private ring of shared memory several columns ahead, so the bytes in flight do
// not cost registers and no barrier is needed (a lane reads only what it copied itself).
//
// The per-cell arithmetic is that of prop.cuh, term by term; cells outside an update's guards get
// a zero coefficient and keep their value.
//
// What bounds it: HBM bandwidth, nearly (4001 x 1601, lean: 257 MB of DRAM traffic in 46.5 us; an
// addition of two arrays into a third takes 48 us for the same 36 bytes per cell), then the latency
// of a warp's own instructions (six cycles each at nine warps per SM).  Measured per forward step:
// 4001 x 1601 with 16-bit strips 70.2 -> 53 us, 3301 x 1501 49.8 -> 40.4, 3001 x 1403 37.9 -> 34.1;
// grids that stay in L2 are faster with the step kernels (2501 x 1203: 24.6 against 25.3 us, 1601 x
// 801: 14.2 against 16.8).
#pragma once
#include "prop.cuh"

namespace swd {

constexpr int MARCH_OWN = 112;   // rows a warp owns of its 128
constexpr int MARCH_LC = 4;

typedef unsigned long long mx2;   // a packed pair of floats

__device__ __forceinline__ mx2 m_fma(mx2 a, mx2 b, mx2 c)
{
    mx2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ mx2 m_dup(float x)
{
    mx2 d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
    return d;
}
struct F4 {   // four rows as two packed pairs
    mx2 a, b;
};
__device__ __forceinline__ float4 m_unpack(F4 v)
{
    float4 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v.a));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.z), "=f"(r.w) : "l"(v.b));
    return r;
}
__device__ __forceinline__ F4 m_pack(float4 v)
{
    F4 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.a) : "f"(v.x), "f"(v.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.b) : "f"(v.z), "f"(v.w));
    return r;
}
__device__ __forceinline__ F4 m_lds(const float *p)
{
    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p);
    return F4{v.x, v.y};
}
// d += c * (x - y), each of the four products rounded as the scalar expression is (x - y is formed
// as fma(y, -1, x), one rounding)
__device__ __forceinline__ void m_tap(F4 &d, mx2 c, F4 x, F4 y, mx2 minus1)
{
    d.a = m_fma(c, m_fma(y.a, minus1, x.a), d.a);
    d.b = m_fma(c, m_fma(y.b, minus1, x.b), d.b);
}

__device__ __forceinline__ void cp16(float *dst, const float *src)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// rows z - 3 .. z - 1 and z + 4 .. z + 7 (P) or z - 4 .. z - 1 and z + 4 .. z + 6 (V) around a lane's four
__device__ __forceinline__ void m_window(float4 o, float w[12])
{
    const unsigned f = 0xffffffffu;
    w[0] = __shfl_up_sync(f, o.x, 1);
    w[1] = __shfl_up_sync(f, o.y, 1);
    w[2] = __shfl_up_sync(f, o.z, 1);
    w[3] = __shfl_up_sync(f, o.w, 1);
    w[4] = o.x; w[5] = o.y; w[6] = o.z; w[7] = o.w;
    w[8] = __shfl_down_sync(f, o.x, 1);
    w[9] = __shfl_down_sync(f, o.y, 1);
    w[10] = __shfl_down_sync(f, o.z, 1);
    w[11] = __shfl_down_sync(f, o.w, 1);
}
// z derivatives: P at half rows (velocity), V at rows (pressure)
__device__ __forceinline__ float4 m_dz_p(const float w[12], const float (&c)[MAXLC])
{
    float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
        for (int ic = 0; ic < MARCH_LC; ic++) el(d, q) += c[ic] * (w[4 + q + ic + 1] - w[4 + q - ic]);
    return d;
}
__device__ __forceinline__ float4 m_dz_v(const float w[12], const float (&c)[MAXLC])
{
    float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
        for (int ic = 0; ic < MARCH_LC; ic++) el(d, q) += c[ic] * (w[4 + q + ic] - w[4 + q - ic - 1]);
    return d;
}
__device__ __forceinline__ float4 m_mask(float4 v, unsigned m)
{
    return make_float4(m & 1 ? v.x : 0.f, m & 2 ? v.y : 0.f, m & 4 ? v.z : 0.f, m & 8 ? v.w : 0.f);
}

// One wavefield of a step: in and out copies; the pressure's CPML memories stay in place.
struct MWave {
    const float *p, *vx, *vz, *ppx, *ppz;
    float *po, *vxo, *vzo, *ppxo, *ppzo;
    float *pvx, *pvz;
};

struct MFwdArgs {
    Geo g;
    Cpml c;
    Mat m;
    MWave w;
    const int *itp;
    int itoff;
    const float *wav0;
    int sx, sz;
    // boundary strips in FP32: the store itself ([nt][slen]), or a ring of MARCH_RING steps that
    // k_march_encode turns into 16-bit codes; nullptr to skip (ring then 1)
    float *strip;
    int slen, ring;
    Wells wells;
    float *seis;        // [r_n][nt], written by the tasks that hold a well column; nullptr to skip
    int nt;
    const int4 *task;   // per warp: first column, columns (a multiple of 8 plus 1), row tile, MARCH_* bits
};

constexpr int MARCH_FRAME = 1;    // not wholly inside the lean box: guards and CPML terms
constexpr int MARCH_XFRAME = 2;   // some column of it has a non-zero x profile
constexpr int MARCH_WELL = 4;     // some column of it is a well
constexpr int MARCH_NARROW = 17;  // columns of a task that touches the frame
constexpr int MARCH_RING = 64;    // steps of FP32 strips kept until they are encoded

// ring depth in columns: six arrays inside the lean box, ten in the frame
constexpr int MARCH_DL = 3, MARCH_DG = 2;
constexpr int MARCH_MAXC = 72;    // columns a task reads at most (C + 7)
// bytes per warp: max(6 * MARCH_DL, 10 * MARCH_DG) columns of 128 floats and the task's x profiles
constexpr int MARCH_FWD_SMEM = 10 * 2 * 512 + 4 * MARCH_MAXC * 4;

template <bool LEAN>
__device__ __forceinline__ void march_fwd(const MFwdArgs &a, float *ring, int x0, int C, bool fx, bool well, int z0)
{
    constexpr int LC = MARCH_LC, NA = LEAN ? 6 : 10, D = LEAN ? MARCH_DL : MARCH_DG;
    const Geo &g = a.g;
    const int lane = threadIdx.x, ntx = g.ntx, ntz = g.ntz, ldz = g.ldz;
    const int zc = min(z0, ldz - 4);   // rows past the array read its last ones (they feed no updated cell)
    const bool own = lane >= 2 && lane < 30 && z0 < ldz;
    const mx2 minus1 = m_dup(-1.f);
    mx2 cx[LC];
#pragma unroll
    for (int i = 0; i < LC; i++) cx[i] = m_dup(g.cx[i]);
    unsigned mp = 15u, mv = 15u;
    float4 az = make_float4(0.f, 0.f, 0.f, 0.f), bz = az, azh = az, bzh = az;
    bool fz = false;
    int zband = 0, zoff = 0, xmid = 0;   // strip rows of this lane: top or bottom band, rows between
    if (!LEAN) {
        mp = mv = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int z = z0 + q;
            if (z >= LC && z <= ntz - LC) mp |= 1u << q;
            if (z >= LC - 1 && z <= ntz - LC - 1) mv |= 1u << q;
        }
        if (z0 >= 0 && z0 < ldz) {
            az = ldg4(a.c.az + z0); bz = ldg4(a.c.bz + z0);
            azh = ldg4(a.c.azh + z0); bzh = ldg4(a.c.bzh + z0);
        }
        if (a.strip) {
            const int nx = ntx - 2 * g.pmlc;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int z = z0 + q;
                if (z < g.pmlc || z > ntz - g.pmlc - 1 || !own) continue;
                if (z < g.pmlc + LC) { zband |= 1 << q; zoff = z0 - g.pmlc; }
                else if (z >= ntz - g.pmlc - LC) { zband |= 1 << q; zoff = LC * nx + z0 - (ntz - g.pmlc - LC); }
                else xmid |= 1 << q;
            }
        }
        fz = __any_sync(0xffffffffu, az.x != 0.f || az.y != 0.f || az.z != 0.f || az.w != 0.f || azh.x != 0.f || azh.y != 0.f || azh.z != 0.f || azh.w != 0.f);
    }
    float *xpr = ring + 10 * 2 * 128;   // axh, bxh, ax, bx of columns j0, j0 + 1, ...
    if (!LEAN && fx) {
        const int n = C + 2 * LC - 1;
        for (int i = lane; i < n; i += 32) {
            const int x = min(max(x0 - LC + i, 0), ntx - 1);
            xpr[i] = __ldg(a.c.axh + x);
            xpr[MARCH_MAXC + i] = __ldg(a.c.bxh + x);
            xpr[2 * MARCH_MAXC + i] = __ldg(a.c.ax + x);
            xpr[3 * MARCH_MAXC + i] = __ldg(a.c.bx + x);
        }
        __syncwarp();
    }
    auto col = [&](int x) { return LEAN ? x : min(max(x, 0), ntx - 1); };
    auto off = [&](int x) { return col(x) * ldz + zc; };
    const int it = *a.itp + a.itoff;
    const int j0 = x0 - LC, nj = C + 2 * LC - 1;
    float *mine = ring + 4 * lane;
    auto issue = [&](int n) {   // the columns iteration n (column j0 + n) reads
        if (n < nj) {
            const int j = j0 + n;
            float *s = mine + (n % D) * NA * 128;
            const int oj = off(j);
            cp16(s, a.w.p + off(j + LC));
            cp16(s + 128, a.w.vx + oj);
            cp16(s + 256, a.m.cbx + oj);
            if (!LEAN && fx && xpr[n] != 0.f) cp16(s + 6 * 128, a.w.ppx + oj);
            if (n >= 2 * LC - 1) {
                const int om = off(j - 3);
                cp16(s + 384, a.w.vz + om);
                cp16(s + 512, a.m.cbz + om);
                cp16(s + 640, a.m.ck + om);
                if (!LEAN) {
                    if (fx && xpr[2 * MARCH_MAXC + n - 3] != 0.f) cp16(s + 7 * 128, a.w.pvx + om);
                    if (fz) {
                        cp16(s + 8 * 128, a.w.ppz + om);
                        cp16(s + 9 * 128, a.w.pvz + om);
                    }
                }
            }
        }
        cp_commit();
    };
#pragma unroll
    for (int n = 0; n < D - 1; n++) issue(n);
    F4 pq[8], vq[8];
#pragma unroll
    for (int i = 0; i < 7; i++) pq[i] = m_pack(ld4(a.w.p + off(j0 - 3 + i)));
    pq[7] = pq[6];
#pragma unroll
    for (int i = 0; i < 8; i++) vq[i] = F4{0, 0};
    // lean: eight columns per trip, so the windows' registers are named by the column; frame: one
    // column per trip and the windows moved along (unrolled, its code exceeds the instruction cache
    // and every column refetches it)
    constexpr int UN = LEAN ? 8 : 1;
#pragma unroll 1
    for (int nb = 0; nb < nj; nb += UN) {
#pragma unroll
        for (int u = 0; u < UN; u++) {
            const int n = nb + u, j = j0 + n, m = j - 3;
            issue(n + D - 1);
            cp_wait<D - 1>();
            const float *s = mine + (n % D) * NA * 128;
            pq[(u + 7) & 7] = m_lds(s);
            // ---- vx(j)
            F4 d{0, 0};
#pragma unroll
            for (int ic = 0; ic < LC; ic++) m_tap(d, cx[ic], pq[(u + 4 + ic) & 7], pq[(u + 3 - ic) & 7], minus1);
            if (LEAN) {
                const F4 cb = m_lds(s + 256), v = m_lds(s + 128);
                vq[u].a = m_fma(cb.a, d.a, v.a);
                vq[u].b = m_fma(cb.b, d.b, v.b);
            } else {
                float4 dd = m_unpack(d), cb = ld4(s + 256), v = ld4(s + 128);
                const float ax = fx ? xpr[n] : 0.f;
                if (ax != 0.f) {
                    const float bx = xpr[MARCH_MAXC + n];
                    float4 f = ld4(s + 6 * 128);
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        el(f, q) = bx * elc(f, q) + ax * elc(dd, q);
                        el(dd, q) = elc(dd, q) + elc(f, q);
                    }
                    if (own && j >= x0 && j < x0 + C && j < ntx) st4(a.w.ppxo + off(j), f);
                }
                cb = m_mask(cb, j >= LC - 1 && j <= ntx - LC - 1 ? mp : 0u);
#pragma unroll
                for (int q = 0; q < 4; q++) el(v, q) = elc(cb, q) * elc(dd, q) + elc(v, q);
                vq[u] = m_pack(v);
            }
            if (own && j >= x0 && j < x0 + C && (LEAN || j < ntx)) *reinterpret_cast<ulonglong2 *>(a.w.vxo + off(j)) = make_ulonglong2(vq[u].a, vq[u].b);
            if (n >= 2 * LC - 1) {
            // ---- vz(m), p(m)
            const float4 pm = m_unpack(pq[u]);
            float w[12];
            m_window(pm, w);
            float4 e = m_dz_p(w, g.cz), cz = ld4(s + 512), vz = ld4(s + 384), kc = ld4(s + 640);
            if (!LEAN) {
                if (fz) {
                    float4 f = ld4(s + 8 * 128);
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        el(f, q) = elc(azh, q) != 0.f ? elc(bzh, q) * elc(f, q) + elc(azh, q) * elc(e, q) : 0.f;
                        el(e, q) = elc(e, q) + elc(f, q);
                    }
                    if (own && m < ntx) st4(a.w.ppzo + off(m), f);
                }
                cz = m_mask(cz, m >= LC && m <= ntx - LC ? mv : 0u);
                kc = m_mask(kc, m >= LC && m <= ntx - LC ? mp : 0u);
            }
#pragma unroll
            for (int q = 0; q < 4; q++) el(vz, q) = elc(cz, q) * elc(e, q) + elc(vz, q);
            m_window(vz, w);
            e = m_dz_v(w, g.cz);
            d = F4{0, 0};
#pragma unroll
            for (int ic = 0; ic < LC; ic++) m_tap(d, cx[ic], vq[(u + 5 + ic) & 7], vq[(u + 4 - ic) & 7], minus1);
            float4 dd = m_unpack(d), p = pm;
            if (!LEAN) {
                const float ax = fx ? xpr[2 * MARCH_MAXC + n - 3] : 0.f;
                if (ax != 0.f) {
                    const float bx = xpr[3 * MARCH_MAXC + n - 3];
                    float4 f = ld4(s + 7 * 128);
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        el(f, q) = bx * elc(f, q) + ax * elc(dd, q);
                        el(dd, q) = elc(dd, q) + elc(f, q);
                    }
                    if (own && m < ntx) st4(a.w.pvx + off(m), f);
                }
                float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
                if (fz) {
                    f = ld4(s + 9 * 128);
#pragma unroll
                    for (int q = 0; q < 4; q++) el(f, q) = elc(az, q) != 0.f ? elc(bz, q) * elc(f, q) + elc(az, q) * elc(e, q) : 0.f;
                    if (own && m < ntx) st4(a.w.pvz + off(m), f);
                }
#pragma unroll
                for (int q = 0; q < 4; q++) el(p, q) = elc(kc, q) * (elc(dd, q) + elc(e, q) + elc(f, q)) + elc(p, q);
            } else {
#pragma unroll
                for (int q = 0; q < 4; q++) el(p, q) = elc(kc, q) * (elc(dd, q) + elc(e, q)) + elc(p, q);
            }
            if (m == a.sx && a.sz >= z0 && a.sz < z0 + 4) {
                const float wv = a.wav0[it];
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (a.sz == z0 + q) el(p, q) += wv;
            }
            if (own && (LEAN || m < ntx)) {
                st4(a.w.vzo + off(m), vz);
                st4(a.w.po + off(m), p);
                if (well) {
                    const int wc = __ldg(a.wells.wcol + m);
                    if (wc >= 0) {
                        const int4 tr = __ldg(reinterpret_cast<const int4 *>(a.wells.wmap + (size_t)wc * ldz + z0));
                        const int t[4] = {tr.x, tr.y, tr.z, tr.w};
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (t[q] >= 0 && z0 + q < ntz) a.seis[(size_t)t[q] * a.nt + it] = elc(p, q);
                    }
                }
                if (!LEAN && m >= g.pmlc && m <= ntx - g.pmlc - 1) {
                    float *sp = a.strip + (size_t)(it % a.ring) * a.slen;
                    const int nx = ntx - 2 * g.pmlc, nzs = ntz - 2 * g.pmlc - 2 * LC;
                    if (zband) {
                        float *t = sp + zoff + (m - g.pmlc) * LC;
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (zband >> q & 1) t[q] = elc(p, q);
                    }
                    int xs = -1;   // left or right band: its column
                    if (m < g.pmlc + LC) xs = m - g.pmlc;
                    else if (m >= ntx - g.pmlc - LC) xs = LC + m - (ntx - g.pmlc - LC);
                    if (xs >= 0 && xmid) {
                        float *t = sp + 2 * LC * nx + xs * nzs + (z0 - g.pmlc - LC);
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (xmid >> q & 1) t[q] = elc(p, q);
                    }
                }
            }
            }
            if (!LEAN) {
                const F4 t = vq[0];
#pragma unroll
                for (int i = 0; i < 7; i++) {
                    pq[i] = pq[i + 1];
                    vq[i] = vq[i + 1];
                }
                vq[7] = t;
            }
        }
    }
}

__global__ void __launch_bounds__(32, 16) k_march_fwd(const MFwdArgs a)
{
    extern __shared__ float4 mring4[];
    const int4 t = __ldg(a.task + blockIdx.x);
    const int z0 = t.z * MARCH_OWN - 8 + 4 * (int)threadIdx.x;
    if (t.w & MARCH_FRAME) march_fwd<false>(a, (float *)mring4, t.x, t.y, (t.w & MARCH_XFRAME) != 0, (t.w & MARCH_WELL) != 0, z0);
    else march_fwd<true>(a, (float *)mring4, t.x, t.y, false, (t.w & MARCH_WELL) != 0, z0);
}

// 16-bit strips of up to MARCH_RING steps from their FP32 ring: the codes and block scales k_fwd_p
// would store (one scale per listed 8-column, 128-row block of cell4's grid and step).
// blockIdx.x: block, blockIdx.y: step after *itp + itoff.
struct MEncodeArgs {
    Geo g;
    const float *ringbuf;
    const int *itp;
    int itoff;
    Strips strips;
    const int *list;     // blocks with strip cells: by * gx + bx
    int gx;
};

__global__ void __launch_bounds__(128) k_march_encode(const MEncodeArgs a)
{
    const Geo &g = a.g;
    const int it = *a.itp + a.itoff + blockIdx.y;
    const float *src = a.ringbuf + (size_t)(it % MARCH_RING) * a.strips.slen;
    // one row per thread over the block's eight columns
    const int slot = __ldg(a.list + blockIdx.x), x0 = slot / a.gx * 8, z = slot % a.gx * 128 + threadIdx.x;
    int si[8];
    float p[8], v = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        si[k] = z < g.ntz && x0 + k < g.ntx ? strip_index(x0 + k, z, g.ntx, g.ntz, g.pmlc, MARCH_LC) : -1;
        p[k] = si[k] >= 0 ? src[si[k]] : 0.f;
        v = fmaxf(v, fabsf(p[k]));
    }
    __shared__ float smax[4];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = v;
    __syncthreads();
    const float mx = fmaxf(fmaxf(smax[0], smax[1]), fmaxf(smax[2], smax[3])), inv = enc16_inv(mx);
    if (threadIdx.x == 0) a.strips.scale[(size_t)it * a.strips.nscale + slot] = mx;
#pragma unroll
    for (int k = 0; k < 8; k++)
        if (si[k] >= 0) ((unsigned short *)a.strips.buf)[(size_t)it * a.strips.slen + si[k]] = enc16(p[k], mx, inv, a.strips.prec);
}

}  // namespace swd
