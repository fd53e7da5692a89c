// Dense, matrix-free Helmholtz kernels on the triangle midpoints.
//
//   boundary  C_i = sum_{j != i} A_ij(kappa) B_j     BoundaryOperatorKernel.cl:5-239
//             A_ij = c1 e^{i k r}/r + (c2 (z.mu_j) - c3 (z.nu_i)) (i k r - 1) e^{i k r}/r^3,
//             z = y_j - x_i, r = |z|; c1..c3 already carry 1/(4 pi).
//   near field  the same sum with c3 = 0 at arbitrary points x_i, no pair
//             excluded                               NearFieldOperatorKernel.cl:5-194
//   far field F_i = sum_j (c1 - i k c2 (x_i.mu_j)) e^{-i k x_i.y_j} B_j     FarFieldOperatorKernel.cl:85-133
//   Herglotz  C_i = sum_j (c1 - i k c2 (nu_i.d_j)) e^{-i k x_i.d_j} conj(g_j) HerglotzWaveKernel.cl:85-160
//   incident  plane / radial waves at the midpoints                          IncidentWaveKernel_*.hpp
//
// Plain form (this file; dense64.cu has the FP64 form): a thread owns one or two
// targets and a group of COLS (<= 16) right-hand-side columns of one wave chunk,
// accumulating COLS complex sums per target in registers; a CTA of 128 threads
// streams the sources through shared memory in tiles (midpoint, normal and the
// tile's RHS rows), so every generated kernel entry is reused for COLS complex
// FMAs.  Padded sources are zero (no reading of padded rows, unlike the
// reference's far-field and Herglotz kernels whose mask is always 1,
// FarFieldOperatorKernel.cl:89).
#include "ops.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace baemm
{

namespace
{

template <class R> struct Prm;
template <> struct Prm<float> { using type = ChunkParamsF; };
template <> struct Prm<double> { using type = ChunkParamsD; };

__device__ __forceinline__ void dsincos(float x, float *s, float *c) { __sincosf(x, s, c); }
__device__ __forceinline__ void dsincos(double x, double *s, double *c) { sincos(x, s, c); }
__device__ __forceinline__ void acc_sincos(float x, float *s, float *c) { sincosf(x, s, c); }
__device__ __forceinline__ void acc_sincos(double x, double *s, double *c) { sincos(x, s, c); }

constexpr int kTargets = 128;   // threads per CTA (one target per thread per pass)
constexpr int kTile = 64;       // sources per shared-memory tile

template <class R, int COLS>
struct Tile
{
    R y[kTile][4];
    R mu[kTile][4];
    cplx<R> B[kTile][COLS];
};

// Stage sources [j0, j0 + kTile) of (pos4, aux4) and COLS columns of rows of
// X (ld) starting at column col0.  Out-of-range sources are zero.
template <class R, int COLS, bool AUX, bool CONJ, class Tx>
__device__ __forceinline__ void stage_tile(Tile<R, COLS> &t, const R *__restrict__ pos4, const R *__restrict__ aux4,
                                           const Tx *__restrict__ X, int64_t ldx, int col0, int j0, int nsrc)
{
    const int tid = threadIdx.x;
    if (tid < kTile)
    {
        const int j = j0 + tid;
        #pragma unroll
        for (int d = 0; d < 4; ++d) t.y[tid][d] = (j < nsrc) ? pos4[4 * (int64_t)j + d] : R(0);
    }
    else if (AUX && tid < 2 * kTile)
    {
        const int s = tid - kTile, j = j0 + s;
        #pragma unroll
        for (int d = 0; d < 4; ++d) t.mu[s][d] = (j < nsrc) ? aux4[4 * (int64_t)j + d] : R(0);
    }
    for (int idx = tid; idx < kTile * COLS; idx += kTargets)
    {
        const int s = idx / COLS, k = idx - s * COLS, j = j0 + s;
        cplx<R> v;
        v.x = R(0);
        v.y = R(0);
        if (j < nsrc)
        {
            const Tx b = X[(int64_t)j * ldx + col0 + k];
            v.x = (R)b.x;
            v.y = CONJ ? -(R)b.y : (R)b.y;
        }
        t.B[s][k] = v;
    }
}

// Packed FP32x2 arithmetic (sm_100 FFMA2), one target per thread and the 16
// columns of one wave chunk (variant 1).  A complex MAC  c += a b  is two
// packed FMAs:
//     c += (a.re, a.re) * (b.re, b.im)
//     c += (a.im, a.im) * (-b.im, b.re)
// so the tile stages every RHS row twice, as b and as the swapped, negated
// (-b.im, b.re).
constexpr int kPackedCols = 16;

struct PackedTile
{
    float4 y[kTile];
    float4 mu[kTile];
    float2 B[kTile][kPackedCols];
    float2 Bw[kTile][kPackedCols];
};

template <bool SL, bool DL, bool ADL>
__global__ void __launch_bounds__(kTargets, 4)
boundary_packed_kernel(DenseTargets<float> tg, const float *__restrict__ mid4, const float *__restrict__ nrm4,
                       const float2 *__restrict__ B, float2 *__restrict__ C, const ChunkParamsF *__restrict__ prm,
                       int n, int wc, int wcs)
{
    __shared__ PackedTile tile;
    const int col0 = blockIdx.y * kPackedCols;
    const int ch = col0 / wcs;
    const float kap = prm[ch].kappa;
    const float2 c1 = prm[ch].c[1], c2 = prm[ch].c[2], c3 = prm[ch].c[3];
    const int tid = threadIdx.x;
    const int ti = blockIdx.x * kTargets + tid;
    const int tself = tg.self ? tg.off + ti : -1;
    float3 x = make_float3(0.f, 0.f, 0.f), nu = x;
    if (ti < tg.m)
    {
        const float4 m = reinterpret_cast<const float4 *>(tg.pts4)[ti];
        x = make_float3(m.x, m.y, m.z);
        if (ADL)
        {
            const float4 q = reinterpret_cast<const float4 *>(nrm4)[tg.off + ti];
            nu = make_float3(q.x, q.y, q.z);
        }
    }
    float2 acc[kPackedCols], tacc[kPackedCols];   // running total, this tile's sum (two-level sum)
    #pragma unroll
    for (int k = 0; k < kPackedCols; ++k) acc[k] = make_float2(0.f, 0.f);

    for (int j0 = 0; j0 < n; j0 += kTile)
    {
        __syncthreads();
        if (tid < kTile)
        {
            const int j = j0 + tid;
            tile.y[tid] = (j < n) ? reinterpret_cast<const float4 *>(mid4)[j] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        else if (DL && tid < 2 * kTile)
        {
            const int sidx = tid - kTile, j = j0 + sidx;
            tile.mu[sidx] = (j < n) ? reinterpret_cast<const float4 *>(nrm4)[j] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        for (int idx = tid; idx < kTile * kPackedCols; idx += kTargets)
        {
            const int sidx = idx / kPackedCols, k = idx % kPackedCols, j = j0 + sidx;
            const float2 b = (j < n) ? B[(int64_t)j * wc + col0 + k] : make_float2(0.f, 0.f);
            tile.B[sidx][k] = b;
            tile.Bw[sidx][k] = make_float2(-b.y, b.x);
        }
        __syncthreads();
        const int smax = min(kTile, n - j0);
        #pragma unroll
        for (int k = 0; k < kPackedCols; ++k) tacc[k] = make_float2(0.f, 0.f);
        for (int s = 0; s < smax; ++s)
        {
            const float4 yv = tile.y[s];
            float4 mv = make_float4(0.f, 0.f, 0.f, 0.f);
            if (DL) mv = tile.mu[s];
            const float zx = yv.x - x.x, zy = yv.y - x.y, zz = yv.z - x.z;
            const float r2 = zx * zx + zy * zy + zz * zz;
            const float rinv = (j0 + s == tself) ? 0.f : rsqrtf(r2);
            const float r = r2 * rinv;
            const float kr = kap * r;
            float sn, cs;
            __sincosf(kr, &sn, &cs);
            float ax = 0.f, ay = 0.f;
            if (SL)
            {
                const float er = cs * rinv, ei = sn * rinv;
                ax = c1.x * er - c1.y * ei;
                ay = c1.x * ei + c1.y * er;
            }
            if (DL || ADL)
            {
                const float r3 = rinv * rinv * rinv;
                const float g0 = -(kr * sn + cs) * r3;
                const float g1 = (kr * cs - sn) * r3;
                float fx = 0.f, fy = 0.f;
                if (DL)
                {
                    const float dm = zx * mv.x + zy * mv.y + zz * mv.z;
                    fx += c2.x * dm;
                    fy += c2.y * dm;
                }
                if (ADL)
                {
                    const float dn = zx * nu.x + zy * nu.y + zz * nu.z;
                    fx -= c3.x * dn;
                    fy -= c3.y * dn;
                }
                ax += fx * g0 - fy * g1;
                ay += fx * g1 + fy * g0;
            }
            const float2 Ar = make_float2(ax, ax), Ai = make_float2(ay, ay);
            #pragma unroll
            for (int k = 0; k < kPackedCols; ++k)
            {
                tacc[k] = __ffma2_rn(Ar, tile.B[s][k], tacc[k]);
                tacc[k] = __ffma2_rn(Ai, tile.Bw[s][k], tacc[k]);
            }
        }
        #pragma unroll
        for (int k = 0; k < kPackedCols; ++k) acc[k] = __fadd2_rn(acc[k], tacc[k]);
    }
    if (ti < tg.m)
    {
        float2 *out = &C[(int64_t)ti * wc + col0];
        #pragma unroll
        for (int k = 0; k < kPackedCols; ++k) out[k] = acc[k];
    }
}

// Plain FP32 form over pairs of targets (the default, and variant 2): the two
// halves of every FP32x2 register are two targets (i, i + 128) of the thread, in
// the entry evaluation as well as in the contraction
//     (c.re, c.im) += (a.re b.re - a.im b.im, a.re b.im + a.im b.re),
// four packed FMAs per column and pair of targets, with the right-hand side
// staged as broadcast pairs (b.re, b.re, b.im, b.im): one 16-byte shared load
// per column, no register shuffling, and the entry (about 22 packed
// instructions with the real / imaginary coefficients of the solves, RI) is
// shared by both targets.  Bound by the FP32 pipe: 64 packed FMAs per source
// and pair of targets at 16 columns, a packed FMA taking two of its cycles.
// Each 32-source tile is summed into fresh accumulators and added to running
// totals in shared memory (a private float4 per thread and column; the error of
// one long FP32 chain over ~1e5 sources would be ~5x larger), which leaves the
// registers for four CTAs of 128 threads per SM.
// Measured: 2.80 ms on 20234 triangles x 32 columns (SL + DL', FP32 pipe 72 %
// busy), one target per thread and unpacked FMAs 4.95 ms; 157 us on 5120 x 16 in
// chunks of 8 columns, 480 us before.
constexpr int kPairTile = 32;

template <int COLS>
struct PairTile
{
    float4 g[kPairTile][3];        // (y.x, y.x, y.y, y.y), (y.z, y.z, mu.x, mu.x), (mu.y, mu.y, mu.z, mu.z)
    float4 b[kPairTile][COLS];
    float4 tot[COLS][kTargets];    // (re, re', im, im') of the thread's two targets
};

template <int COLS, bool SL, bool DL, bool ADL, bool RI>
__global__ void __launch_bounds__(kTargets, 4)
boundary_pair_kernel(DenseTargets<float> tg, const float *__restrict__ mid4, const float *__restrict__ nrm4,
                     const float2 *B, float2 *__restrict__ C, const ChunkParamsF *__restrict__ prm,
                     int n, int wc, int wcs, int per_split)
{
    chain_wait();
    __shared__ PairTile<COLS> tile;
    const int tid = threadIdx.x;
    const int col0 = blockIdx.y * COLS;
    const int jb = blockIdx.z * per_split, je = min(n, jb + per_split);   // this split's sources
    const ChunkParamsF &q = prm[col0 / wcs];
    const float2 nk = make_float2(-q.kappa, -q.kappa);
    const float2 c1x = make_float2(q.c[1].x, q.c[1].x), c1y = make_float2(q.c[1].y, q.c[1].y);
    const float2 nc2x = make_float2(-q.c[2].x, -q.c[2].x), nc2y = make_float2(-q.c[2].y, -q.c[2].y);
    const float2 c3x = make_float2(q.c[3].x, q.c[3].x), c3y = make_float2(q.c[3].y, q.c[3].y);
    const int t0 = blockIdx.x * (2 * kTargets) + tid, t1 = t0 + kTargets;
    const int self0 = tg.self ? tg.off + t0 : -1, self1 = tg.self ? tg.off + t1 : -1;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 xa = t0 < tg.m ? reinterpret_cast<const float4 *>(tg.pts4)[t0] : zero;
    const float4 xb = t1 < tg.m ? reinterpret_cast<const float4 *>(tg.pts4)[t1] : zero;
    const float2 nx0 = make_float2(-xa.x, -xb.x), nx1 = make_float2(-xa.y, -xb.y), nx2 = make_float2(-xa.z, -xb.z);
    float2 tn0 = make_float2(0.f, 0.f), tn1 = tn0, tn2 = tn0;
    if (ADL)
    {
        const float4 na = t0 < tg.m ? reinterpret_cast<const float4 *>(nrm4)[tg.off + t0] : zero;
        const float4 nb = t1 < tg.m ? reinterpret_cast<const float4 *>(nrm4)[tg.off + t1] : zero;
        tn0 = make_float2(na.x, nb.x); tn1 = make_float2(na.y, nb.y); tn2 = make_float2(na.z, nb.z);
    }
    #pragma unroll
    for (int k = 0; k < COLS; ++k) tile.tot[k][tid] = zero;   // private to the thread: no barrier needed

    for (int j0 = jb; j0 < je; j0 += kPairTile)
    {
        __syncthreads();
        if (tid < kPairTile)
        {
            const int j = j0 + tid;
            const float4 y = j < je ? reinterpret_cast<const float4 *>(mid4)[j] : zero;
            const float4 mu = DL && j < je ? reinterpret_cast<const float4 *>(nrm4)[j] : zero;
            tile.g[tid][0] = make_float4(y.x, y.x, y.y, y.y);
            tile.g[tid][1] = make_float4(y.z, y.z, mu.x, mu.x);
            tile.g[tid][2] = make_float4(mu.y, mu.y, mu.z, mu.z);
        }
        #pragma unroll
        for (int idx = tid; idx < kPairTile * COLS; idx += kTargets)
        {
            const int s = idx / COLS, k = idx % COLS, j = j0 + s;
            const float2 b = j < je ? B[(int64_t)j * wc + col0 + k] : make_float2(0.f, 0.f);
            tile.b[s][k] = make_float4(b.x, b.x, b.y, b.y);
        }
        __syncthreads();
        const int smax = min(kPairTile, je - j0);
        float2 cr[COLS], ci[COLS];
        #pragma unroll
        for (int k = 0; k < COLS; ++k) cr[k] = ci[k] = make_float2(0.f, 0.f);
        for (int s = 0; s < smax; ++s)
        {
            const float4 ga = tile.g[s][0], gb = tile.g[s][1], gc = tile.g[s][2];
            const float2 zx = __fadd2_rn(make_float2(ga.x, ga.y), nx0);
            const float2 zy = __fadd2_rn(make_float2(ga.z, ga.w), nx1);
            const float2 zz = __fadd2_rn(make_float2(gb.x, gb.y), nx2);
            const float2 r2 = __ffma2_rn(zz, zz, __ffma2_rn(zy, zy, __fmul2_rn(zx, zx)));
            const float2 ri = make_float2(j0 + s == self0 ? 0.f : rsqrtf(r2.x), j0 + s == self1 ? 0.f : rsqrtf(r2.y));
            const float2 nkr = __fmul2_rn(nk, __fmul2_rn(r2, ri));   // -k r
            float sa, ca, sb, cb;
            __sincosf(nkr.x, &sa, &ca);
            __sincosf(nkr.y, &sb, &cb);
            const float2 cs = make_float2(ca, cb), nsn = make_float2(sa, sb);   // cos(k r), -sin(k r)
            // h = c1 / r + u + i k r (-u),  u = -(c2 (z.mu) - c3 (z.nu)) / r^3;  A = e^{i k r} h
            float2 ux = make_float2(0.f, 0.f), uy = ux, hx = ux, hy = ux;
            if (DL || ADL)
            {
                const float2 ri3 = __fmul2_rn(__fmul2_rn(ri, ri), ri);
                if (DL)
                {
                    const float2 dm = __fmul2_rn(
                        __ffma2_rn(zz, make_float2(gc.z, gc.w),
                                   __ffma2_rn(zy, make_float2(gc.x, gc.y), __fmul2_rn(zx, make_float2(gb.z, gb.w)))),
                        ri3);
                    ux = __fmul2_rn(nc2x, dm);
                    if (!RI) uy = __fmul2_rn(nc2y, dm);
                }
                if (ADL)
                {
                    const float2 dn = __fmul2_rn(__ffma2_rn(zz, tn2, __ffma2_rn(zy, tn1, __fmul2_rn(zx, tn0))), ri3);
                    ux = DL ? __ffma2_rn(c3x, dn, ux) : __fmul2_rn(c3x, dn);
                    if (!RI) uy = DL ? __ffma2_rn(c3y, dn, uy) : __fmul2_rn(c3y, dn);
                }
                hx = ux;
                hy = __fmul2_rn(nkr, ux);
                if (!RI)
                {
                    hx = __ffma2_rn(make_float2(-nkr.x, -nkr.y), uy, hx);
                    hy = __fadd2_rn(hy, uy);
                }
            }
            if (SL)
            {
                if (!RI) hx = __ffma2_rn(c1x, ri, hx);
                hy = __ffma2_rn(c1y, ri, hy);
            }
            // (ar, ai) = (hx cos - hy sin, hx sin + hy cos)
            const float2 ar = __ffma2_rn(hy, nsn, __fmul2_rn(hx, cs));
            const float2 ai = __ffma2_rn(hy, cs, __fmul2_rn(make_float2(-hx.x, -hx.y), nsn));
            const float2 nai = make_float2(-ai.x, -ai.y);
            #pragma unroll
            for (int k = 0; k < COLS; ++k)
            {
                const float4 b = tile.b[s][k];
                const float2 br = make_float2(b.x, b.y), bi = make_float2(b.z, b.w);
                cr[k] = __ffma2_rn(ar, br, cr[k]);
                cr[k] = __ffma2_rn(nai, bi, cr[k]);
                ci[k] = __ffma2_rn(ar, bi, ci[k]);
                ci[k] = __ffma2_rn(ai, br, ci[k]);
            }
        }
        #pragma unroll
        for (int k = 0; k < COLS; ++k)
        {
            float4 t = tile.tot[k][tid];
            t.x += cr[k].x; t.y += cr[k].y; t.z += ci[k].x; t.w += ci[k].y;
            tile.tot[k][tid] = t;
        }
    }
    chain_next();
    // with a cluster of S parts of the sources, block r adds columns r, r + S, ... of all of them in order
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    if (S > 1) cluster.sync();
    float2 *out = C + (int64_t)(blockIdx.z / S) * tg.m * wc + col0;
    for (int k = rank; k < COLS; k += S)
    {
        float4 t = S > 1 ? *cluster.map_shared_rank(&tile.tot[k][tid], 0) : tile.tot[k][tid];
        for (int q = 1; q < S; ++q)
        {
            const float4 v = *cluster.map_shared_rank(&tile.tot[k][tid], q);
            t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
        }
        if (t0 < tg.m) out[(int64_t)t0 * wc + k] = make_float2(t.x, t.z);
        if (t1 < tg.m) out[(int64_t)t1 * wc + k] = make_float2(t.y, t.w);
    }
    if (S > 1) cluster.sync();   // no block leaves while its totals are read
}

// C = the sum of the partial blocks of a split launch, in order (four loads in flight).
template <class R>
__global__ void split_sum_kernel(const cplx<R> *partial, int splits, int64_t elems, cplx<R> *__restrict__ C)
{
    chain_begin();
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= elems) return;
    const cplx<R> *p = partial + e;
    cplx<R> s = p[0];
    int q = 1;
    for (; q + 4 <= splits; q += 4)
    {
        cplx<R> v[4];
        #pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = p[(q + u) * elems];
        #pragma unroll
        for (int u = 0; u < 4; ++u) { s.x += v[u].x; s.y += v[u].y; }
    }
    for (; q < splits; ++q)
    {
        const cplx<R> v = p[q * elems];
        s.x += v.x;
        s.y += v.y;
    }
    C[e] = s;
}

template <class R, int COLS, bool SL, bool DL>
__global__ void __launch_bounds__(kTargets)
farfield_partial_kernel(const R *__restrict__ meas4, const R *__restrict__ mid4, const R *__restrict__ nrm4,
                        const cplx<R> *__restrict__ B, const typename Prm<R>::type *__restrict__ prm, int m, int n,
                        int wc, int wcs, int per_split, cplx<R> *__restrict__ partial)
{
    __shared__ Tile<R, COLS> tile;
    const int i = blockIdx.x * kTargets + threadIdx.x;
    const int col0 = blockIdx.y * COLS;
    const int split = blockIdx.z;
    const int ch = col0 / wcs;
    const R kap = prm[ch].kappa;
    const cplx<R> c1 = prm[ch].c[1], c2 = prm[ch].c[2];
    R x0 = R(0), x1 = R(0), x2 = R(0);
    if (i < m) { x0 = meas4[4 * (int64_t)i]; x1 = meas4[4 * (int64_t)i + 1]; x2 = meas4[4 * (int64_t)i + 2]; }
    cplx<R> acc[COLS];
    #pragma unroll
    for (int k = 0; k < COLS; ++k) { acc[k].x = R(0); acc[k].y = R(0); }
    const int jb = split * per_split, je = min(n, jb + per_split);
    for (int j0 = jb; j0 < je; j0 += kTile)
    {
        __syncthreads();
        stage_tile<R, COLS, DL, false>(tile, mid4, nrm4, B, wc, col0, j0, je);
        __syncthreads();
        const int smax = min(kTile, je - j0);
        for (int s = 0; s < smax; ++s)
        {
            const R th = kap * (tile.y[s][0] * x0 + tile.y[s][1] * x1 + tile.y[s][2] * x2);
            R sn, cs;
            dsincos(th, &sn, &cs);
            // e = exp(-i th); A = (c1 + c2 (-i k mu.x)) e
            cplx<R> f;
            f.x = SL ? c1.x : R(0);
            f.y = SL ? c1.y : R(0);
            if (DL)
            {
                const R dk = kap * (tile.mu[s][0] * x0 + tile.mu[s][1] * x1 + tile.mu[s][2] * x2);
                f.x += c2.y * dk;
                f.y -= c2.x * dk;
            }
            cplx<R> A;
            A.x = f.x * cs + f.y * sn;
            A.y = f.y * cs - f.x * sn;
            #pragma unroll
            for (int k = 0; k < COLS; ++k) cfma(acc[k], A, tile.B[s][k]);
        }
    }
    if (i < m)
    {
        cplx<R> *out = &partial[((int64_t)split * m + i) * wc + col0];
        #pragma unroll
        for (int k = 0; k < COLS; ++k) out[k] = acc[k];
    }
}

// Sum of the splits' partial blocks in double, times alpha, plus beta C.  One
// block per 32 elements: 8 rows of threads take every eighth split each (four
// loads in flight), added in row order.  (One thread per element over all
// splits: 42 us for 148 x 256 x 32 double values, now 3.3 us for 74.)
constexpr int kReduceRows = 8;
template <class R>
__global__ void __launch_bounds__(32 * kReduceRows)
farfield_reduce_kernel(const cplx<R> *partial, int splits, int m, int wc, double2 alpha, double2 beta,
                       double2 *Cout, int64_t ldC)
{
    chain_begin();
    __shared__ double2 row[kReduceRows][32];
    const int64_t elems = (int64_t)m * wc, idx = (int64_t)blockIdx.x * 32 + threadIdx.x;
    double2 t = make_double2(0.0, 0.0);
    if (idx < elems)
    {
        #pragma unroll 4
        for (int s = threadIdx.y; s < splits; s += kReduceRows)
        {
            const cplx<R> p = partial[s * elems + idx];
            t.x += (double)p.x;
            t.y += (double)p.y;
        }
    }
    row[threadIdx.y][threadIdx.x] = t;
    __syncthreads();
    if (threadIdx.y != 0 || idx >= elems) return;
    #pragma unroll
    for (int s = 1; s < kReduceRows; ++s)
    {
        t.x += row[s][threadIdx.x].x;
        t.y += row[s][threadIdx.x].y;
    }
    const int64_t i = idx / wc;
    double2 o = make_double2(alpha.x * t.x - alpha.y * t.y, alpha.x * t.y + alpha.y * t.x);
    double2 *c = &Cout[i * ldC + (idx - i * wc)];
    if (beta.x != 0.0 || beta.y != 0.0)
    {
        const double2 b = *c;
        o.x += beta.x * b.x - beta.y * b.y;
        o.y += beta.x * b.y + beta.y * b.x;
    }
    *c = o;
}

template <class R, int COLS, bool SL, bool DL>
__global__ void __launch_bounds__(kTargets)
herglotz_kernel(const R *__restrict__ mid4, const R *__restrict__ nrm4, const R *__restrict__ meas4,
                const double2 *__restrict__ g, int64_t ldg, const typename Prm<R>::type *__restrict__ prm, int n, int m,
                int wc, int wcs, cplx<R> *__restrict__ C)
{
    __shared__ Tile<R, COLS> tile;
    const int i = blockIdx.x * kTargets + threadIdx.x;
    const int col0 = blockIdx.y * COLS;
    const int ch = col0 / wcs;
    const R kap = prm[ch].kappa;
    const cplx<R> c1 = prm[ch].c[1], c2 = prm[ch].c[2];
    R x0 = R(0), x1 = R(0), x2 = R(0), n0 = R(0), n1 = R(0), n2 = R(0);
    if (i < n)
    {
        x0 = mid4[4 * (int64_t)i]; x1 = mid4[4 * (int64_t)i + 1]; x2 = mid4[4 * (int64_t)i + 2];
        n0 = nrm4[4 * (int64_t)i]; n1 = nrm4[4 * (int64_t)i + 1]; n2 = nrm4[4 * (int64_t)i + 2];
    }
    cplx<R> acc[COLS];
    #pragma unroll
    for (int k = 0; k < COLS; ++k) { acc[k].x = R(0); acc[k].y = R(0); }
    for (int j0 = 0; j0 < m; j0 += kTile)
    {
        __syncthreads();
        stage_tile<R, COLS, false, true>(tile, meas4, nullptr, g, ldg, col0, j0, m);
        __syncthreads();
        const int smax = min(kTile, m - j0);
        for (int s = 0; s < smax; ++s)
        {
            const R th = kap * (tile.y[s][0] * x0 + tile.y[s][1] * x1 + tile.y[s][2] * x2);
            R sn, cs;
            dsincos(th, &sn, &cs);
            cplx<R> f;
            f.x = SL ? c1.x : R(0);
            f.y = SL ? c1.y : R(0);
            if (DL)
            {
                const R dk = kap * (n0 * tile.y[s][0] + n1 * tile.y[s][1] + n2 * tile.y[s][2]);
                f.x += c2.y * dk;
                f.y -= c2.x * dk;
            }
            cplx<R> A;
            A.x = f.x * cs + f.y * sn;
            A.y = f.y * cs - f.x * sn;
            #pragma unroll
            for (int k = 0; k < COLS; ++k) cfma(acc[k], A, tile.B[s][k]);
        }
    }
    if (i < n)
    {
        cplx<R> *out = &C[(int64_t)i * wc + col0];
        #pragma unroll
        for (int k = 0; k < COLS; ++k) out[k] = acc[k];
    }
}

template <class R>
__global__ void incident_kernel(int64_t nt, const R *__restrict__ mid4, const R *__restrict__ nrm4,
                                const typename Prm<R>::type *__restrict__ prm, int wc, int wcs,
                                const R *__restrict__ dirs, int type, cplx<R> *__restrict__ C)
{
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nt * wc) return;
    const int64_t i = idx / wc;
    const int k = (int)(idx - i * wc);
    const int ch = k / wcs, j = k - ch * wcs;
    const R K = prm[ch].kappa;
    const cplx<R> c1 = prm[ch].c[1], c2 = prm[ch].c[2];
    const R m0 = mid4[4 * i], m1 = mid4[4 * i + 1], m2 = mid4[4 * i + 2];
    const R q0 = nrm4[4 * i], q1 = nrm4[4 * i + 1], q2 = nrm4[4 * i + 2];
    const R d0 = dirs[3 * j], d1 = dirs[3 * j + 1], d2 = dirs[3 * j + 2];
    cplx<R> f, e;
    if (type == BAEMM_WAVE_RADIAL)
    {
        // IncidentWaveKernel_Radial.hpp:28-51
        const R oofp = R(1) / (R(2) * (R(2) * R(3.14159265358979323846)));
        const R dl0 = m0 - d0, dl1 = m1 - d1, dl2 = m2 - d2;
        const R R2 = dl0 * dl0 + dl1 * dl1 + dl2 * dl2;
        const R Rr = sqrt(R2), oR = R(1) / Rr, oR2 = R(1) / R2;
        const R dn = q0 * dl0 + q1 * dl1 + q2 * dl2;
        const R A = oofp * oR;
        cplx<R> Bc;
        Bc.x = -dn * oR2;
        Bc.y = dn * K * oR;
        // factor = c1 A + c2 A B
        f.x = c1.x * A + A * (c2.x * Bc.x - c2.y * Bc.y);
        f.y = c1.y * A + A * (c2.x * Bc.y + c2.y * Bc.x);
        R s, c;
        acc_sincos(K * Rr, &s, &c);
        e.x = c;
        e.y = s;
    }
    else
    {
        // IncidentWaveKernel_Plane.hpp:208-227: (c1 + c2 i k <d,n>) e^{i k <d,x>}
        const R dm = m0 * d0 + m1 * d1 + m2 * d2;
        const R dn = q0 * d0 + q1 * d1 + q2 * d2;
        f.x = c1.x - c2.y * (K * dn);
        f.y = c1.y + c2.x * (K * dn);
        R s, c;
        acc_sincos(K * dm, &s, &c);
        e.x = c;
        e.y = s;
    }
    C[idx] = cmul(f, e);
}

// Evaluation points (m x 3 doubles) as m x 4 reals, w = 0
// (ApplyNearFieldOperators.hpp:96-107 pads them the same way).
template <class R>
__global__ void pack_points_kernel(int64_t m, const double *pts3, R *__restrict__ pts4)
{
    chain_begin();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    pts4[4 * i + 0] = (R)pts3[3 * i + 0];
    pts4[4 * i + 1] = (R)pts3[3 * i + 1];
    pts4[4 * i + 2] = (R)pts3[3 * i + 2];
    pts4[4 * i + 3] = R(0);
}

// ---- dispatch helpers -----------------------------------------------------------
// The kernel template KERNEL<ARGS..., SL, DL, ADL> of an operator code
#define BAEMM_BY_LAYERS(LAUNCH)                     \
    switch (code)                                   \
    {                                               \
        case 1: LAUNCH(true, false, false); break;  \
        case 2: LAUNCH(false, true, false); break;  \
        case 3: LAUNCH(true, true, false); break;   \
        case 4: LAUNCH(false, false, true); break;  \
        case 5: LAUNCH(true, false, true); break;   \
        case 6: LAUNCH(false, true, true); break;   \
        case 7: LAUNCH(true, true, true); break;    \
        default: break;                             \
    }

template <class R, int COLS>
void farfield_cols(const OpFlags &f, dim3 grid, cudaStream_t st, const R *meas, const R *mid, const R *nrm,
                   const cplx<R> *B, const typename Prm<R>::type *p, int m, int n, int wc, int wcs, int per_split,
                   cplx<R> *partial)
{
    if (f.sl() && f.dl())
        farfield_partial_kernel<R, COLS, true, true><<<grid, kTargets, 0, st>>>(meas, mid, nrm, B, p, m, n, wc, wcs, per_split, partial);
    else if (f.sl())
        farfield_partial_kernel<R, COLS, true, false><<<grid, kTargets, 0, st>>>(meas, mid, nrm, B, p, m, n, wc, wcs, per_split, partial);
    else
        farfield_partial_kernel<R, COLS, false, true><<<grid, kTargets, 0, st>>>(meas, mid, nrm, B, p, m, n, wc, wcs, per_split, partial);
}

template <class R, int COLS>
void herglotz_cols(const OpFlags &f, dim3 grid, cudaStream_t st, const R *mid, const R *nrm, const R *meas,
                   const double2 *g, int64_t ldg, const typename Prm<R>::type *p, int n, int m, int wc, int wcs,
                   cplx<R> *C)
{
    if (f.sl() && f.dl())
        herglotz_kernel<R, COLS, true, true><<<grid, kTargets, 0, st>>>(mid, nrm, meas, g, ldg, p, n, m, wc, wcs, C);
    else if (f.sl())
        herglotz_kernel<R, COLS, true, false><<<grid, kTargets, 0, st>>>(mid, nrm, meas, g, ldg, p, n, m, wc, wcs, C);
    else
        herglotz_kernel<R, COLS, false, true><<<grid, kTargets, 0, st>>>(mid, nrm, meas, g, ldg, p, n, m, wc, wcs, C);
}

template <class R> const R *geo_mid(const MeshDev &m);
template <> const float *geo_mid<float>(const MeshDev &m) { return m.mid_f; }
template <> const double *geo_mid<double>(const MeshDev &m) { return m.mid_d; }
template <class R> const R *geo_nrm(const MeshDev &m);
template <> const float *geo_nrm<float>(const MeshDev &m) { return m.nrm_f; }
template <> const double *geo_nrm<double>(const MeshDev &m) { return m.nrm_d; }
template <class R> const R *geo_meas(const MeshDev &m);
template <> const float *geo_meas<float>(const MeshDev &m) { return m.meas_f; }
template <> const double *geo_meas<double>(const MeshDev &m) { return m.meas_d; }

inline int cols_for(int wcs) { return wcs < 16 ? wcs : 16; }

void packed_dispatch(int code, dim3 grid, cudaStream_t st, DenseTargets<float> tg, const float *mid, const float *nrm,
                     const float2 *B, float2 *C, const ChunkParamsF *p, int n, int wc, int wcs)
{
#define BAEMM_PK(SL, DL, ADL) \
    boundary_packed_kernel<SL, DL, ADL><<<grid, kTargets, 0, st>>>(tg, mid, nrm, B, C, p, n, wc, wcs)
    BAEMM_BY_LAYERS(BAEMM_PK)
#undef BAEMM_PK
}

template <int COLS, bool RI>
void pair_dispatch(int code, dim3 grid, int cluster, cudaStream_t st, DenseTargets<float> tg, const float *mid,
                   const float *nrm, const float2 *B, float2 *C, const ChunkParamsF *p, int n, int wc, int wcs,
                   int per_part)
{
#define BAEMM_PR(SL, DL, ADL) \
    launch_chained(boundary_pair_kernel<COLS, SL, DL, ADL, RI>, grid, kTargets, 0, st, cluster, tg, mid, nrm, B, C, p, \
                     n, wc, wcs, per_part)
    BAEMM_BY_LAYERS(BAEMM_PR)
#undef BAEMM_PR
}

// Room (elements) for partial blocks at `at`.  A stream under capture grows
// nothing: an allocation would end its capture.
template <class R>
size_t partial_room(SplitSpace<R> ws, size_t capacity, cudaStream_t st, cplx<R> *&at)
{
    at = ws.fixed;
    if (!ws.grow) return std::min(ws.elems, capacity);
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (ws.grow->n < capacity)
    {
        BAEMM_CUDA(cudaStreamIsCapturing(st, &capture));
        if (capture == cudaStreamCaptureStatusNone) try
        {
            ws.grow->reserve(capacity);
        }
        catch (const Error &)   // no memory: not split
        {
        }
    }
    at = ws.grow->p;
    return std::min(ws.grow->n, capacity);   // the split does not depend on what else the context has run
}

// Ctri (tg.m x wc) = K Btri over all nt sources for the targets tg, of which the
// context's launches have up to most_targets.
template <class R>
void dense_dispatch(const MeshDev &m, const OpFlags &f, const void *chunk_params, int wc, int wcs,
                    DenseTargets<R> tg, int64_t most_targets, const cplx<R> *Btri, cplx<R> *Ctri, cudaStream_t st,
                    int variant, SplitSpace<R> ws)
{
    if (!f.any_layer() || m.nt == 0 || tg.m == 0) return;
    BAEMM_REQUIRE(wcs >= 1 && wcs <= 64 && (wcs & (wcs - 1)) == 0, BAEMM_ERR_SIZE,
                  "wave_chunk_size must be a power of two <= 64");
    const int n = (int)m.nt;
    const int cols = cols_for(wcs);
    const int code = (f.sl() ? 1 : 0) | (f.dl() ? 2 : 0) | (f.adl() ? 4 : 0);
    const auto *p = static_cast<const typename Prm<R>::type *>(chunk_params);
    const R *mid = geo_mid<R>(m), *nrm = geo_nrm<R>(m);
    const int64_t elems = (int64_t)tg.m * wc;
    const size_t capacity = split_capacity(n, most_targets * wc, sizeof(cplx<R>));
    SourceSplit split;
    cplx<R> *out = nullptr;
    if constexpr (std::is_same<R, double>::value)
    {
        const size_t room = partial_room<R>(ws, capacity, st, out);
        split = dense_split(d64_ctas(d64_unit(wc, wcs), tg.m, wc), n, tc_sm_count(), room / elems);
        launch_boundary_d64(m, f, p, wc, wcs, tg, Btri, split.blocks > 1 ? out : Ctri, split, st);
    }
    else
    {
        if (variant == 1 && cols == kPackedCols)
        {
            const dim3 grid(ceil_div(tg.m, kTargets), wc / cols);
            packed_dispatch(code, grid, st, tg, mid, nrm, Btri, Ctri, p, n, wc, wcs);
        }
        else
        {
            dim3 pairs(ceil_div(tg.m, 2 * kTargets), wc / cols);
            const size_t room = partial_room<R>(ws, capacity, st, out);
            split = dense_split((int64_t)pairs.x * pairs.y, n, tc_sm_count(), room / elems);
            pairs.z = split.parts();
            const int per_part = ceil_div(n, split.parts());
            cplx<R> *dst = split.blocks > 1 ? out : Ctri;
            // single layer imaginary, double layers real (the tuples of the solves): RI
            const bool ri = !f.re_sl && !f.im_dl && !f.im_adl;
#define BAEMM_PC(COLS) \
    ri ? pair_dispatch<COLS, true>(code, pairs, split.cluster, st, tg, mid, nrm, Btri, dst, p, n, wc, wcs, per_part) \
       : pair_dispatch<COLS, false>(code, pairs, split.cluster, st, tg, mid, nrm, Btri, dst, p, n, wc, wcs, per_part)
            if (cols == 16) BAEMM_PC(16);
            else if (cols == 8) BAEMM_PC(8);
            else if (cols == 4) BAEMM_PC(4);
            else if (cols == 2) BAEMM_PC(2);
            else BAEMM_PC(1);
#undef BAEMM_PC
        }
        BAEMM_LAUNCH_CHECK();
    }
    if (split.blocks > 1)
    {
        launch_chained(split_sum_kernel<R>, ceil_div(elems, 256), 256, 0, st, 1, out, split.blocks, elems, Ctri);
        BAEMM_LAUNCH_CHECK();
    }
}

} // namespace

// The split with the least estimated time,
//     (n / parts + kSplitCost) * max(ceil(ctas parts / SMs), 2) [+ kSumCost if blocks > 1]:
// the sources of one CTA times the CTAs of the busiest SM.  An SM needs about two
// CTAs of four warps before its pipe is shared rather than idle (hence the 2); a
// CTA costs about kSplitCost sources to start, drain and sum, and the sum of
// partial blocks (one more kernel) about kSumCost.  Without a split a launch of a
// few CTAs leaves most SMs idle, and one of 1.1 CTAs per SM runs at half speed.
// Two parts share a cluster: larger ones leave SMs unevenly loaded (5120 x 16
// host apply: 268 us without clusters, 250 with clusters of 2, 327 of 8; far
// field of 81920 triangles in 256 directions x 32: 288, 285, 441).  Up to
// kTiny sources one cluster takes all parts: its kernel is slower (320 x 16:
// 13.2 instead of 7.3 + 3.1 us with its sum) but saves a launch, which is what
// such a call waits for (27.3 instead of 29.4 us a call).
constexpr int kTiny = 512, kMinSources = 16, kCluster = 2, kMostBlocks = 64;
SourceSplit dense_split(int64_t ctas, int64_t n, int sms, int64_t most_blocks)
{
    constexpr int kSplitCost = 24, kSumCost = 70;
    const int cluster = n <= kTiny ? 8 : kCluster;
    const int most = n <= kTiny ? 8 : kCluster * (int)std::max<int64_t>(1, std::min<int64_t>(kMostBlocks, most_blocks));
    SourceSplit best;
    double best_cost = 0.0;
    for (int parts = 1; parts <= most && (parts == 1 || n >= (int64_t)parts * kMinSources); parts += parts < cluster ? 1 : cluster)
    {
        const double per_sm = (double)std::max<int64_t>((ctas * parts + sms - 1) / sms, 2);
        const double cost = ((double)n / parts + (parts > 1 ? kSplitCost : 0)) * per_sm + (parts > cluster ? kSumCost : 0);
        if (parts == 1 || cost < 0.97 * best_cost)
        {
            best.cluster = std::min(parts, cluster);
            best.blocks = parts / best.cluster;
            best_cost = cost;
        }
    }
    return best;
}

// At most kMostBlocks blocks of at least kCluster * kMinSources sources; 16 MB of
// them (which give a launch of few CTAs the whole chip) or kEvenBlocks (which even
// out the waves of a launch that has more); and beyond 64 MB no more than four, up
// to 1 GB.  Without these limits the split takes up to 14 blocks of a large result;
// of 17000 random shapes 100 would want more than they leave, for a gain of 3.0 to
// 3.6 % by the estimate above.
size_t split_capacity(int64_t n, int64_t elems, size_t elem_bytes)
{
    constexpr size_t MB = (size_t)1 << 20, kEvenBlocks = 20, kLargeBlocks = 4;
    if (n <= kTiny) return 0;
    const size_t blocks = std::min<int64_t>(kMostBlocks, n / (kCluster * kMinSources)), e = (size_t)elems;
    const size_t most = std::min(std::max(64 * MB / elem_bytes, kLargeBlocks * e), 1024 * MB / elem_bytes);
    return std::min({blocks * e, std::max(16 * MB / elem_bytes, kEvenBlocks * e), most});
}

template <class R>
void launch_boundary_dense(const MeshDev &m, const OpFlags &f, const void *chunk_params, int wc, int wcs,
                           const cplx<R> *Btri, cplx<R> *Ctri, cudaStream_t st, SplitSpace<R> ws, int variant,
                           int64_t row_begin, int64_t row_end)
{
    const int64_t r0 = std::max<int64_t>(0, row_begin), r1 = row_end < 0 ? m.nt : std::min<int64_t>(row_end, m.nt);
    if (r1 <= r0) return;
    dense_dispatch<R>(m, f, chunk_params, wc, wcs, DenseTargets<R>{geo_mid<R>(m) + 4 * r0, (int)(r1 - r0), 1, (int)r0},
                      m.nt, Btri, Ctri + r0 * wc, st, variant, ws);
}

template <class R>
void launch_nearfield_dense(const MeshDev &m, const OpFlags &f, const void *chunk_params, int wc, int wcs,
                            const R *pts4, int64_t npts, const cplx<R> *Btri, cplx<R> *Cpts, cudaStream_t st,
                            SplitSpace<R> ws, int variant)
{
    BAEMM_REQUIRE(!f.adl() && !f.mass(), BAEMM_ERR_ARG, "near field: single and double layer only");
    BAEMM_REQUIRE(npts <= INT32_MAX, BAEMM_ERR_SIZE, "too many evaluation points");
    dense_dispatch<R>(m, f, chunk_params, wc, wcs, DenseTargets<R>{pts4, (int)npts, 0, 0}, npts, Btri, Cpts, st, variant,
                      ws);
}

template <class R>
void launch_pack_points(int64_t m, const double *pts3, R *pts4, cudaStream_t st)
{
    if (m == 0) return;
    launch_chained(pack_points_kernel<R>, ceil_div(m, 256), 256, 0, st, 1, m, pts3, pts4);
    BAEMM_LAUNCH_CHECK();
}

// The FP32 far field's parts of whole tiles, four CTAs per SM
constexpr int kFarCtas = 4 * 148;
static int farfield_splits(const MeshDev &m, int wc, int wcs)
{
    const int ctas = ceil_div(m.nm, kTargets) * (wc / cols_for(wcs));
    return std::max(1, std::min(ceil_div(kFarCtas, ctas), ceil_div(m.nt, kTile)));
}

size_t farfield_partial_elems(const MeshDev &m, int wc, bool fp64)
{
    const size_t elems = (size_t)m.nm * wc;
    if (fp64) return std::max(elems, split_capacity(m.nt, (int64_t)elems, sizeof(double2)));
    // at most kFarCtas / CTAs + 1 parts, a CTA's results at most kTargets x 16
    return std::min(elems * ceil_div(m.nt, kTile), elems + (size_t)kFarCtas * kTargets * 16);
}

template <class R>
void launch_farfield(const MeshDev &m, const OpFlags &f, const void *chunk_params, int wc, int wcs,
                     const cplx<R> *Btri, cplx<R> *partial, size_t partial_cap, double2 alpha, double2 beta,
                     double2 *Cout, int64_t ldC, cudaStream_t st)
{
    if (!(f.sl() || f.dl()) || m.nm == 0) return;
    BAEMM_REQUIRE(wcs >= 1 && wcs <= 64 && (wcs & (wcs - 1)) == 0, BAEMM_ERR_SIZE,
                  "wave_chunk_size must be a power of two <= 64");
    constexpr bool fp64 = std::is_same<R, double>::value;
    const size_t room = partial_cap / ((size_t)m.nm * wc);   // blocks of results
    BAEMM_REQUIRE(room >= 1, BAEMM_ERR_SIZE, "far-field partial buffer too small");
    SourceSplit split;
    const auto *p = static_cast<const typename Prm<R>::type *>(chunk_params);
    const int mm = (int)m.nm, n = (int)m.nt;
    if constexpr (fp64)
    {
        const size_t most = farfield_partial_elems(m, wc, true) / ((size_t)m.nm * wc);
        split = dense_split(d64_ctas(d64_unit(wc, wcs), m.nm, wc), m.nt, tc_sm_count(), std::min(room, most));
        launch_farfield_d64(m, f, p, wc, wcs, Btri, partial, split, st);
    }
    else
    {
        split.blocks = (int)std::min<size_t>(farfield_splits(m, wc, wcs), room);
        const int cols = cols_for(wcs);
        const int per_split = ceil_div(ceil_div(n, split.blocks), kTile) * kTile;
        split.blocks = ceil_div(n, per_split);
        const dim3 grid(ceil_div(m.nm, kTargets), wc / cols, split.blocks);
        const R *mid = geo_mid<R>(m), *nrm = geo_nrm<R>(m), *meas = geo_meas<R>(m);
        switch (cols)
        {
            case 1: farfield_cols<R, 1>(f, grid, st, meas, mid, nrm, Btri, p, mm, n, wc, wcs, per_split, partial); break;
            case 2: farfield_cols<R, 2>(f, grid, st, meas, mid, nrm, Btri, p, mm, n, wc, wcs, per_split, partial); break;
            case 4: farfield_cols<R, 4>(f, grid, st, meas, mid, nrm, Btri, p, mm, n, wc, wcs, per_split, partial); break;
            case 8: farfield_cols<R, 8>(f, grid, st, meas, mid, nrm, Btri, p, mm, n, wc, wcs, per_split, partial); break;
            default: farfield_cols<R, 16>(f, grid, st, meas, mid, nrm, Btri, p, mm, n, wc, wcs, per_split, partial); break;
        }
        BAEMM_LAUNCH_CHECK();
    }
    launch_chained(farfield_reduce_kernel<R>, ceil_div((int64_t)mm * wc, 32), dim3(32, kReduceRows), 0, st, 1, partial,
                   split.blocks, mm, wc, alpha, beta, Cout, ldC);
    BAEMM_LAUNCH_CHECK();
}

template <class R>
void launch_herglotz(const MeshDev &m, const OpFlags &f, const void *chunk_params, int wc, int wcs, const double2 *g,
                     int64_t ldg, cplx<R> *Ctri, cudaStream_t st)
{
    if (!(f.sl() || f.dl()) || m.nt == 0) return;
    const int cols = cols_for(wcs);
    dim3 grid(ceil_div(m.nt, kTargets), wc / cols);
    const auto *p = static_cast<const typename Prm<R>::type *>(chunk_params);
    const R *mid = geo_mid<R>(m), *nrm = geo_nrm<R>(m), *meas = geo_meas<R>(m);
    const int n = (int)m.nt, mm = (int)m.nm;
    switch (cols)
    {
        case 1: herglotz_cols<R, 1>(f, grid, st, mid, nrm, meas, g, ldg, p, n, mm, wc, wcs, Ctri); break;
        case 2: herglotz_cols<R, 2>(f, grid, st, mid, nrm, meas, g, ldg, p, n, mm, wc, wcs, Ctri); break;
        case 4: herglotz_cols<R, 4>(f, grid, st, mid, nrm, meas, g, ldg, p, n, mm, wc, wcs, Ctri); break;
        case 8: herglotz_cols<R, 8>(f, grid, st, mid, nrm, meas, g, ldg, p, n, mm, wc, wcs, Ctri); break;
        case 16: herglotz_cols<R, 16>(f, grid, st, mid, nrm, meas, g, ldg, p, n, mm, wc, wcs, Ctri); break;
        default: throw Error(BAEMM_ERR_SIZE, "wave_chunk_size must be a power of two <= 64");
    }
    BAEMM_LAUNCH_CHECK();
}

template <class R>
void launch_incident(const MeshDev &m, const void *chunk_params, int wc, int wcs, const R *dirs, int type,
                     cplx<R> *Ctri, cudaStream_t st)
{
    const int64_t n = m.nt * wc;
    if (n == 0) return;
    incident_kernel<R><<<ceil_div(n, 256), 256, 0, st>>>(m.nt, geo_mid<R>(m), geo_nrm<R>(m),
                                                         static_cast<const typename Prm<R>::type *>(chunk_params), wc,
                                                         wcs, dirs, type, Ctri);
    BAEMM_LAUNCH_CHECK();
}

template void launch_boundary_dense<float>(const MeshDev &, const OpFlags &, const void *, int, int, const float2 *,
                                           float2 *, cudaStream_t, SplitSpace<float>, int, int64_t, int64_t);
template void launch_pack_points<float>(int64_t, const double *, float *, cudaStream_t);
template void launch_pack_points<double>(int64_t, const double *, double *, cudaStream_t);
template void launch_nearfield_dense<float>(const MeshDev &, const OpFlags &, const void *, int, int, const float *,
                                            int64_t, const float2 *, float2 *, cudaStream_t, SplitSpace<float>, int);
template void launch_nearfield_dense<double>(const MeshDev &, const OpFlags &, const void *, int, int, const double *,
                                             int64_t, const double2 *, double2 *, cudaStream_t, SplitSpace<double>, int);
template void launch_boundary_dense<double>(const MeshDev &, const OpFlags &, const void *, int, int, const double2 *,
                                            double2 *, cudaStream_t, SplitSpace<double>, int, int64_t, int64_t);
template void launch_farfield<float>(const MeshDev &, const OpFlags &, const void *, int, int, const float2 *, float2 *,
                                     size_t, double2, double2, double2 *, int64_t, cudaStream_t);
template void launch_farfield<double>(const MeshDev &, const OpFlags &, const void *, int, int, const double2 *,
                                      double2 *, size_t, double2, double2, double2 *, int64_t, cudaStream_t);
template void launch_herglotz<float>(const MeshDev &, const OpFlags &, const void *, int, int, const double2 *, int64_t,
                                     float2 *, cudaStream_t);
template void launch_herglotz<double>(const MeshDev &, const OpFlags &, const void *, int, int, const double2 *,
                                      int64_t, double2 *, cudaStream_t);
template void launch_incident<float>(const MeshDev &, const void *, int, int, const float *, int, float2 *,
                                     cudaStream_t);
template void launch_incident<double>(const MeshDev &, const void *, int, int, const double *, int, double2 *,
                                      cudaStream_t);

} // namespace baemm
