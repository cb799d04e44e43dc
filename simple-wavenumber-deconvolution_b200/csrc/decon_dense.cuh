// decon_dense.cuh -- the deconvolution's windows as small real matrix products.
//
// The window's transforms have L = filterwin + psfwin - 1 points per axis (odd, prime for the
// usual geometries), but only filterwin (image patch) or psfwin (PSF) of them are non-zero and
// only outwin of the results are read.  Both patches are odd-sized, so indices are taken from the
// patch's centre, t = -h .. h, and each axis splits into an even and an odd part:
//   ee(t1,t2) = a(t1,t2) + a(t1,-t2) + a(-t1,t2) + a(-t1,-t2),  eo, oe, oo with the signs of the
//   odd axes, for t1, t2 >= 0 (an axis value of 0 counts once).
// The four parts transform by real cosine and sine tables (C[t][k] = cos(2 pi t k / L), S sin):
//   X_ee = C^T ee C,  X_eo = C^T eo S,  X_oe = S^T oe C,  X_oo = S^T oo S      (k1, k2 >= 0)
//   A^( k1,k2) = (X_ee - X_oo) - i (X_oe + X_eo),   A^(-k1,k2) = (X_ee + X_oo) + i (X_oe - X_eo),
// the remaining quadrants being complex conjugates.  The phases of the three centres (image
// patch at FX/2, PSF at psfwin/2, output at FX/2 - psfwin/2) cancel in M^ conj(S^), so none is
// applied.  With D(k1,k2) = a + ib and D(-k1,k2) = c + id the inverse transform is, again as four
// real products over k1, k2 >= 0,
//   F_ee = 2(a + c), F_oo = 2(c - a), F_eo = -2(b + d), F_oe = -2(b - d)   (halved where k1 is its
//   own negative, and where k2 is),
//   out(+-r1, +-r2) = O_ee +- O_oo +- O_eo +- O_oe,  O_ee = C F_ee C^T, ...
// That is about a quarter of the operations of the dense complex products, and on 227-point
// windows (129^2 patch, 127^2 output: 21 MFLOP) fewer than the chirp-z FFTs of 512 points execute,
// at the rate of register-tiled FMAs instead of that of shuffles.
//
// k_dense_psf transforms each PSF that some window uses (lattice points; every window's own blend
// with psf_interp) once and keeps S^(k1,k2), S^(-k1,k2) and max|S^|^2 in global memory;
// k_dense_window runs one window per CTA, blk columns k2 at a time: P = part x table, X = table x
// P, the damped division in FP64, and the two inverse products, the last one accumulated over the
// column blocks in registers.
//
// What bounds it: issue and shared-memory reads of one CTA's warps between its barriers (a 227-point
// window needs 82k cycles of FMAs and takes 257k).  Measured per image (window kernel alone; the
// FFT windows before): 4001 x 1601, 227 points: 1.49 ms (14.0); 1601 x 801, 157 points: 0.41 (4.2);
// 845 x 702, 101 points: 0.34 (2.7).  Rows of a thread's tile lie apart, so that neighbouring lanes
// read neighbouring rows on distinct banks (adjacent rows: 0.80 -> 0.59 ms on 450 windows of 227
// points); packed FMAs then 0.59 -> 0.55.
// The L1 norms that scale both patches are double sums (the FFT path forms the reference's serial
// single-precision sums).
#pragma once
#include "decon.cuh"

namespace swd {

// Sizes of one window geometry; axis 1 = x, axis 2 = z.
struct DenseGeo {
    int L1, L2, K1, K2;        // transform lengths, non-negative frequencies
    int hm1, hm2, hp1, hp2;    // half sizes of the image patch and of the PSF
    int ho1, ho2;              // half output window
    int K1p, R1p, R2p;         // K1, ho1 + 1 rounded up to 4, ho2 + 1 rounded up to 8
    int TR1, TR2, KT1, KT2;    // rows and row pitches of the tables (pitch / 4 odd: rows on distinct banks)
    int blk, NB, yp;           // columns k2 per block, blocks, row pitch of a block in shared memory
    int npsf, pz;              // PSFs transformed, lattice points along z (0: one PSF per window)
    int nthr, tiles;           // threads of the window kernel, output tiles per thread
};

__host__ __device__ inline int up4(int v) { return (v + 3) & ~3; }
__host__ __device__ inline int up8(int v) { return (v + 7) & ~7; }
// row pitch >= n, multiple of 4 with an odd quotient
__host__ __device__ inline int odd4(int n) { const int p = up4(n); return (p / 4) & 1 ? p : p + 4; }

__host__ __device__ inline size_t dense_tab1(const DenseGeo &d) { return 2 * (size_t)d.TR1 * d.KT1; }
__host__ __device__ inline size_t dense_tab_len(const DenseGeo &d)
{
    return dense_tab1(d) + (d.L1 == d.L2 ? 0 : 2 * (size_t)d.TR2 * d.KT2);
}
// floats of the parts of a patch with half sizes h1, h2, and of a block's P (or Y) and X
__host__ __device__ inline size_t dense_src(int h1, int h2) { return 4 * (size_t)(h2 + 1) * up4(h1 + 1); }
__host__ __device__ inline size_t dense_p(const DenseGeo &d, int h1)
{
    const size_t p = 4 * (size_t)up4(h1 + 1) * d.yp, y = 4 * (size_t)d.R1p * d.yp;
    return p > y ? p : y;
}
__host__ __device__ inline size_t dense_x(const DenseGeo &d) { return 4 * (size_t)d.K1p * d.yp; }
__host__ __device__ inline size_t dense_smem(const DenseGeo &d, int h1, int h2)
{
    size_t work = dense_src(h1, h2) + dense_p(d, h1) + dense_x(d);
    const size_t out = 4 * (size_t)d.R1p * d.R2p;   // the output parts reuse the work area
    if (work < out) work = out;
    return sizeof(float) * (dense_tab_len(d) + work);
}
__host__ __device__ inline size_t dense_spec(const DenseGeo &d) { return (size_t)d.K1 * (d.NB * d.blk); }   // float4 per PSF

// Shared memory a window's CTA may take, and the limit both kernels are given on every call: it belongs
// to the kernel on the device, not to a context, so no call may lower it under another thread's launch.
constexpr int DENSE_SMEM_MAX = 226 * 1024;

// Tables of one axis: C then S, [TR][KT] each, zero for k >= K; double, rounded once.
__global__ void k_dense_tables(float *t, int L, int K, int TR, int KT)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < TR * KT; i += gridDim.x * blockDim.x) {
        const int r = i / KT, k = i % KT;
        double s = 0.0, c = 0.0;
        if (k < K) sincospi(2.0 * (double)(((long long)r * k) % L) / (double)L, &s, &c);
        t[i] = (float)c;
        t[TR * KT + i] = (float)s;
    }
}

// Packed single-precision pairs (one FMA instruction for two results, each rounded as fmaf rounds)
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 dup2(float x)
{
    f32x2 d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
    return d;
}
__device__ __forceinline__ ulonglong2 ld22(const float *p) { return *reinterpret_cast<const ulonglong2 *>(p); }
__device__ __forceinline__ void st22(float *p, f32x2 a, f32x2 b) { *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(a, b); }

// block-wide sum in double (order fixed by the thread layout); red holds one value per warp
__device__ __forceinline__ double dense_sum(double v, double *red)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += red[w];
    __syncthreads();
    return s;
}

// Even/odd parts of a patch: val(i1, i2), i = -h .. h.  Part p = 2 * (odd in axis 1) + (odd in
// axis 2) at src[p * (h2 + 1) * s1 + t2 * s1 + t1], s1 = up4(h1 + 1).
// PSF (IMAGE false): scaled by its L1 norm, each value divided in double.  Image patch: scaled by
// the power of two below its norm, which rounds nothing and needs no conversions (a division per
// value kept the conversion unit busy for an eighth of the kernel); the remaining factor of the
// normalisation is returned and enters the division in double.  An image norm of at most 1e-15
// counts as 1e-10.
template <bool IMAGE, class V>
__device__ __forceinline__ double dense_split(float *src, int h1, int h2, double *red, V val)
{
    const int s1 = up4(h1 + 1), n = (h2 + 1) * s1;
    double sum = 0.0;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const int t1 = j / (h2 + 1), t2 = j % (h2 + 1);   // t2 fastest: neighbouring image columns
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (t1 <= h1) {
            v[0] = val(t1, t2);
            if (t2 > 0) v[1] = val(t1, -t2);
            if (t1 > 0) v[2] = val(-t1, t2);
            if (t1 > 0 && t2 > 0) v[3] = val(-t1, -t2);
        }
        sum += (double)((fabsf(v[0]) + fabsf(v[1])) + (fabsf(v[2]) + fabsf(v[3])));
#pragma unroll
        for (int p = 0; p < 4; p++) src[p * n + t2 * s1 + t1] = v[p];
    }
    double nrm = dense_sum(sum, red);
    if (IMAGE && nrm <= 1.0e-15) nrm = (double)1.0e-10f;
    float sc = 1.f;
    double rest = 1.0;
    if (IMAGE) {
        const int e = max(-126, min(126, ((__double2hiint(nrm) >> 20) & 0x7ff) - 1023));
        sc = __int_as_float((127 - e) << 23);
        rest = 1.0 / (nrm * (double)sc);
    }
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const int t1 = j / (h2 + 1), t2 = j % (h2 + 1), at = t2 * s1 + t1;
        float v[4];
#pragma unroll
        for (int p = 0; p < 4; p++) v[p] = IMAGE ? src[p * n + at] * sc : (float)((double)src[p * n + at] / nrm);
        if (t1 > h1) v[0] = v[1] = v[2] = v[3] = 0.f;   // padding
        // cells on an axis have no partner there: their absent values stay out of the sums
        const bool q1 = t1 > 0, q2 = t2 > 0;
        const float pm = q2 ? v[1] : 0.f, mp = q1 ? v[2] : 0.f, mm = q1 && q2 ? v[3] : 0.f;
        src[at] = (v[0] + mp) + (pm + mm);
        src[n + at] = q2 ? (v[0] + mp) - (pm + mm) : 0.f;
        src[2 * n + at] = q1 ? (v[0] - mp) + (pm - mm) : 0.f;
        src[3 * n + at] = q1 && q2 ? (v[0] - mp) - (pm - mm) : 0.f;
    }
    __syncthreads();
    return rest;
}

// P[part][t1][k2 of the block] = sum_t2 src[part][t2][t1] T2[t2][k2], 4 x 4 outputs per thread
__device__ __forceinline__ void dense_rows(const DenseGeo &d, const float *src, float *P, const float *T2, int h1, int h2, int kb)
{
    const int s1 = up4(h1 + 1), n1 = s1 / 4, n2 = d.blk / 4, nt = 4 * n1 * n2;
    for (int id = threadIdx.x; id < nt; id += blockDim.x) {
        const int part = id / (n1 * n2), r = id % (n1 * n2), i1 = r / n2, i2 = r % n2;
        const float *a = src + (size_t)part * (h2 + 1) * s1 + 4 * i1;
        const float *t = T2 + (part & 1) * d.TR2 * d.KT2 + kb + 4 * i2;
        f32x2 acc[4][2] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
#pragma unroll 4
        for (int k = 0; k <= h2; k++) {
            const float4 x = ld4(a + k * s1);
            const ulonglong2 y = ld22(t + k * d.KT2);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const f32x2 xx = dup2(elc(x, i));
                acc[i][0] = fma2(xx, y.x, acc[i][0]);
                acc[i][1] = fma2(xx, y.y, acc[i][1]);
            }
        }
        float *o = P + ((size_t)part * s1 + 4 * i1) * d.yp + 4 * i2;
#pragma unroll
        for (int i = 0; i < 4; i++) st22(o + i * d.yp, acc[i][0], acc[i][1]);
    }
    __syncthreads();
}

// X[part][k1][k2 of the block] = sum_t1 T1[t1][k1] P[part][t1][k2], 4 x 8 outputs per thread
__device__ __forceinline__ void dense_cols(const DenseGeo &d, const float *P, float *X, const float *T1, int h1)
{
    const int s1 = up4(h1 + 1), n1 = d.K1p / 4, n2 = d.blk / 8, nt = 4 * n1 * n2;
    for (int id = threadIdx.x; id < nt; id += blockDim.x) {
        const int part = id / (n1 * n2), r = id % (n1 * n2), i1 = r / n2, i2 = r % n2;
        const float *a = T1 + (part >> 1) * d.TR1 * d.KT1 + 4 * i1;
        const float *t = P + (size_t)part * s1 * d.yp + 8 * i2;
        f32x2 acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = 0;
#pragma unroll 4
        for (int k = 0; k <= h1; k++) {
            const float4 x = ld4(a + k * d.KT1);
            const ulonglong2 y0 = ld22(t + k * d.yp), y1 = ld22(t + k * d.yp + 4);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const f32x2 xx = dup2(elc(x, i));
                acc[i][0] = fma2(xx, y0.x, acc[i][0]);
                acc[i][1] = fma2(xx, y0.y, acc[i][1]);
                acc[i][2] = fma2(xx, y1.x, acc[i][2]);
                acc[i][3] = fma2(xx, y1.y, acc[i][3]);
            }
        }
        float *o = X + ((size_t)part * d.K1p + 4 * i1) * d.yp + 8 * i2;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            st22(o + i * d.yp, acc[i][0], acc[i][1]);
            st22(o + i * d.yp + 4, acc[i][2], acc[i][3]);
        }
    }
    __syncthreads();
}

// tables into shared memory; returns the two axes' tables
__device__ __forceinline__ void dense_load_tables(const DenseGeo &d, const float *__restrict__ tabs, float *sm, const float *&T1, const float *&T2)
{
    const int n = (int)dense_tab_len(d);
    for (int j = threadIdx.x; j < n / 4; j += blockDim.x) st4(sm + 4 * j, ldg4(tabs + 4 * j));
    T1 = sm;
    T2 = d.L1 == d.L2 ? sm : sm + dense_tab1(d);
}

// S^ of one PSF: spec[p][k1][k2] = (S^(k1,k2), S^(-k1,k2)), smax[p] = max |S^|^2
__global__ void __launch_bounds__(512) k_dense_psf(DeconGeo g, DenseGeo d, const float *__restrict__ psf, float4 *__restrict__ spec,
                                                   float *__restrict__ smax, const float *__restrict__ tabs)
{
    extern __shared__ float4 dsm4[];
    __shared__ double red[32];
    __shared__ unsigned s_max;
    float *sm = (float *)dsm4;
    const float *T1, *T2;
    dense_load_tables(d, tabs, sm, T1, T2);
    float *src = sm + dense_tab_len(d), *P = src + dense_src(d.hp1, d.hp2), *X = P + dense_p(d, d.hp1);
    if (threadIdx.x == 0) s_max = 0u;
    const int p = blockIdx.x;
    if (d.pz > 0) {   // lattice point (3 + p / pz, 3 + p % pz)
        const int x0 = g.halfpsfwx + (3 + p / d.pz) * g.psfwinx, z0 = g.halfpsfwz + (3 + p % d.pz) * g.psfwinz;
        dense_split<false>(src, d.hp1, d.hp2, red, [&](int a, int b) { return img_at(psf, g.nx, g.nz, x0 + a, z0 + b); });
    } else {          // window p's own PSF: nearest, or the blend of the four around its centre
        const PsfPick q = psf_pick(g, p);
        dense_split<false>(src, d.hp1, d.hp2, red, [&](int a, int b) { return psf_value(g, q, psf, a + d.hp1, b + d.hp2); });
    }
    const int kw = d.NB * d.blk;
    float4 *o = spec + (size_t)p * dense_spec(d);
    float fm = 0.f;
    for (int b = 0; b < d.NB; b++) {
        dense_rows(d, src, P, T2, d.hp1, d.hp2, b * d.blk);
        dense_cols(d, P, X, T1, d.hp1);
        const int xs = d.K1p * d.yp;
        for (int j = threadIdx.x; j < d.K1 * d.blk; j += blockDim.x) {
            const int k1 = j / d.blk, c = j % d.blk, k2 = b * d.blk + c, q = k1 * d.yp + c;
            const float ee = X[q], eo = X[xs + q], oe = X[2 * xs + q], oo = X[3 * xs + q];
            const float4 v = make_float4(ee - oo, -(oe + eo), ee + oo, oe - eo);
            o[(size_t)k1 * kw + k2] = v;
            if (k2 < d.K2) {
                fm = fmaxf(fm, (float)((double)v.x * (double)v.x + (double)v.y * (double)v.y));
                fm = fmaxf(fm, (float)((double)v.z * (double)v.z + (double)v.w * (double)v.w));
            }
        }
        __syncthreads();
    }
    for (int s = 16; s > 0; s >>= 1) fm = fmaxf(fm, __shfl_xor_sync(0xffffffffu, fm, s));
    if ((threadIdx.x & 31) == 0) atomicMax(&s_max, __float_as_uint(fm));
    __syncthreads();
    if (threadIdx.x == 0) smax[p] = __uint_as_float(s_max);
}

// One window per CTA.  NT: output tiles (4 x 8 results) a thread accumulates.
template <int NT>
__global__ void __launch_bounds__(NT == 1 ? 512 : 384) k_dense_window(DeconGeo g, DenseGeo d, const float *__restrict__ mig,
                                                                      const float4 *__restrict__ spec, const float *__restrict__ smax,
                                                                      float *__restrict__ winout, const float *__restrict__ tabs)
{
    extern __shared__ float4 dsm4[];
    __shared__ double red[32];
    float *sm = (float *)dsm4;
    const float *T1, *T2;
    dense_load_tables(d, tabs, sm, T1, T2);
    float *src = sm + dense_tab_len(d), *P = src + dense_src(d.hm1, d.hm2), *X = P + dense_p(d, d.hm1), *Y = P;
    const int w = blockIdx.x, tid = threadIdx.x, nthr = blockDim.x;
    const int ix = g.stepwinx * (w / g.stepnumz), iz = g.stepwinz * (w % g.stepnumz);
    const double rest = dense_split<true>(src, d.hm1, d.hm2, red, [&](int a, int b) {
        const int x = ix + a, z = iz + b;
        return x >= 0 && x < g.nxp && z >= 0 && z < g.nzp ? img_at(mig, g.nx, g.nz, x, z) : 0.f;
    });
    int p = w;
    if (d.pz > 0) {
        const PsfPick q = psf_pick(g, w);
        p = (q.ixf - 3) * d.pz + q.izf - 3;
    }
    const float4 *sp = spec + (size_t)p * dense_spec(d);
    float fft_max = smax[p] * g.epsilon;
    if (fft_max == 0.0f) fft_max = 1.0e-15f;
    // output tiles of this thread: part, 4 rows r1, 8 columns r2
    const int n1 = d.R1p / 4, n2 = d.R2p / 8, ntile = 4 * n1 * n2;
    float acc[NT][4][8];
#pragma unroll
    for (int u = 0; u < NT; u++)
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) acc[u][i][j] = 0.f;
    const int kw = d.NB * d.blk, xs = d.K1p * d.yp;
    for (int b = 0; b < d.NB; b++) {
        dense_rows(d, src, P, T2, d.hm1, d.hm2, b * d.blk);
        dense_cols(d, P, X, T1, d.hm1);
        // damped division (the denominator rounded through float as the reference does), then the
        // four real parts of the inverse
        for (int j = tid; j < d.K1 * d.blk; j += nthr) {
            const int k1 = j / d.blk, c = j % d.blk, k2 = b * d.blk + c, q = k1 * d.yp + c;
            if (k2 >= d.K2) continue;   // X is zero there
            const float4 s = __ldg(sp + (size_t)k1 * kw + k2);
            const double ee = X[q], eo = X[xs + q], oe = X[2 * xs + q], oo = X[3 * xs + q];
            const double mr0 = ee - oo, mi0 = -(oe + eo), mr1 = ee + oo, mi1 = oe - eo;
            const double sr0 = s.x, si0 = s.y, sr1 = s.z, si1 = s.w;
            const double q0 = rest / (double)(float)((sr0 * sr0 + si0 * si0) + (double)fft_max);
            const double q1 = rest / (double)(float)((sr1 * sr1 + si1 * si1) + (double)fft_max);
            const float da = (float)((mr0 * sr0 + mi0 * si0) * q0), db = (float)((mi0 * sr0 - mr0 * si0) * q0);
            const float dc = (float)((mr1 * sr1 + mi1 * si1) * q1), dd = (float)((mi1 * sr1 - mr1 * si1) * q1);
            const float wt = (2 * k1 % d.L1 == 0 ? 1.f : 2.f) * (2 * k2 % d.L2 == 0 ? 0.5f : 1.f);
            X[q] = wt * (da + dc);
            X[xs + q] = -wt * (db + dd);
            X[2 * xs + q] = -wt * (db - dd);
            X[3 * xs + q] = wt * (dc - da);
        }
        __syncthreads();
        // Y[part][r1][k2] = sum_k1 T1[r1][k1] F[part][k1][k2], 4 x 4 outputs per thread
        for (int id = tid; id < 4 * n1 * (d.blk / 4); id += nthr) {
            const int m2 = d.blk / 4, part = id / (n1 * m2), r = id % (n1 * m2), i1 = r / m2, i2 = r % m2;
            // the thread's rows lie n1 apart, so neighbouring lanes read neighbouring rows (distinct banks)
            const float *t = T1 + (part >> 1) * d.TR1 * d.KT1 + i1 * d.KT1;
            const int rs = n1 * d.KT1;
            const float *f = X + (size_t)part * xs + 4 * i2;
            f32x2 y[4][2] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
            for (int k = 0; k < d.K1p; k += 4) {
                float4 a[4];
                ulonglong2 e[4];
#pragma unroll
                for (int i = 0; i < 4; i++) a[i] = ld4(t + i * rs + k);
#pragma unroll
                for (int i = 0; i < 4; i++) e[i] = ld22(f + (k + i) * d.yp);
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const f32x2 aa = dup2(elc(a[i], q));
                        y[i][0] = fma2(aa, e[q].x, y[i][0]);
                        y[i][1] = fma2(aa, e[q].y, y[i][1]);
                    }
            }
            float *o = Y + ((size_t)part * d.R1p + i1) * d.yp + 4 * i2;
#pragma unroll
            for (int i = 0; i < 4; i++) st22(o + i * n1 * d.yp, y[i][0], y[i][1]);
        }
        __syncthreads();
        // out[part][r1][r2] += sum_k2 Y[part][r1][k2] T2[r2][k2]
#pragma unroll
        for (int u = 0; u < NT; u++) {
            const int id = tid + u * nthr;
            if (id < ntile) {
                const int part = id / (n1 * n2), r = id % (n1 * n2), i1 = r / n2, i2 = r % n2;
                const float *a = Y + ((size_t)part * d.R1p + i1) * d.yp;
                const float *t = T2 + (part & 1) * d.TR2 * d.KT2 + i2 * d.KT2 + b * d.blk;
                const int as = n1 * d.yp, ts = n2 * d.KT2;
                for (int k = 0; k < d.blk; k += 4) {
                    float4 x[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) x[i] = ld4(a + i * as + k);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const float4 y = ld4(t + j * ts + k);
#pragma unroll
                        for (int q = 0; q < 4; q++)
#pragma unroll
                            for (int i = 0; i < 4; i++) acc[u][i][j] = fmaf(elc(x[i], q), elc(y, q), acc[u][i][j]);
                    }
                }
            }
        }
        __syncthreads();
    }
    // the four parts to shared memory, then their signed sums to the window's slot
    float *O = src;
    const int os = d.R1p * d.R2p;
#pragma unroll
    for (int u = 0; u < NT; u++) {
        const int id = tid + u * nthr;
        if (id < ntile) {
            const int part = id / (n1 * n2), r = id % (n1 * n2), i1 = r / n2, i2 = r % n2;
            float *o = O + (size_t)part * os + i1 * d.R2p + i2;
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) o[i * n1 * d.R2p + j * n2] = acc[u][i][j];
        }
    }
    __syncthreads();
    const int nout = g.outwinx * g.outwinz;
    float *out = winout + (size_t)w * nout;
    for (int j = tid; j < nout; j += nthr) {
        const int r1 = j / g.outwinz - d.ho1, r2 = j % g.outwinz - d.ho2;
        const int at = abs(r1) * d.R2p + abs(r2);
        const float ee = O[at], eo = O[os + at], oe = O[2 * os + at], oo = O[3 * os + at];
        const float s1 = r1 < 0 ? -1.f : 1.f, s2 = r2 < 0 ? -1.f : 1.f;
        out[j] = (ee + s2 * eo) + s1 * (oe + s2 * oo);
    }
}

}  // namespace swd
