// FP64 form of the dense kernels on the FP64 matrix instructions (sm_100a).
//
//   boundary / near field   A_ij as in dense.cu, targets the midpoints or points
//   far field               A_ij = (c1 - i k c2 (x_i.mu_j)) e^{-i k x_i.y_j}
//
// Both are C = A B with kernel entries A computed on the fly.  A warp owns 16
// targets and up to 32 columns; per step of 8 sources every thread evaluates
// the four entries that mma.m16n8k8 wants in its A registers (targets g, g + 8,
// sources t, t + 4 of the step; g = lane / 4, t = lane % 4), so an entry goes
// from the arithmetic into the matrix instruction without passing through
// shared memory.  The right-hand sides are staged in the order of the B
// registers (one 16-byte load per thread and 8 columns).
//
// The FP64 pipe bounds it: matrix and scalar FP64 instructions share it (37
// TFLOP/s by either, and the mix takes the sum of both times), so what counts
// is the number of FP64 operations per entry:
//   * the geometry of a pair is shared by the E wavenumbers of a work unit, the
//     entry by all columns of its wavenumber;
//   * coefficients of the solves (single layer imaginary, double layers real:
//     RI) need one rotation per entry;
//   * sine and cosine share one argument reduction; 1/r is the hardware's
//     approximation and one third-order step.
// The complex product is four real ones, Re C = Re A Re B - Im A Im B and
// Im C = Re A Im B + Im A Re B, each part accumulated by itself.  (Three products,
// P1 = Re A Re B, P2 = Im A Im B, P3 = (Re A + Im A)(Re B + Im B), need 48 multiply-
// adds per entry and 16 columns instead of 64, 22.2 instead of 24.9 ms below, but
// round the smaller part against the larger: at kappa = 1e-8 the imaginary part of
// a single-layer apply was off by 4e-9 of itself, now by 1e-15.)
// Sums over at most kSegment sources (and the splits of small launches) are added
// to running totals in shared memory.
// Measured: 24.9 ms on 41666 triangles x 32 columns (two wavenumbers, SL + DL;
// 3.47e9 entries at 39 FP64 instructions and 64 matrix multiply-adds: 78 % of
// the pipe), 41.6 ms with scalar FMAs; far field of 81920 triangles in 256
// directions x 32 columns 319 us, 437 before; 1280 x 32 43 us, 446 before
// (unsplit).  Three blocks per SM (168 registers) take 24.9 ms, 460 and 57 us;
// staging element by element instead of in register order cost 4 ms in bank
// conflicts.
#include "ops.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

namespace baemm
{
namespace
{

constexpr int kThreads = 128;             // 4 warps
constexpr int kWarpTargets = 16;          // rows of the matrix instruction
constexpr int kStage = 32;                // sources per shared-memory stage
constexpr int kSegment = 512;             // sources summed in registers before they go to the totals

// sin and cos of x, |x| < 1e5: Cody and Waite's reduction by multiples
// of pi/2 in two parts (the first difference is exact, the second part carries
// the next 53 bits), then the Taylor polynomials on [-pi/4, pi/4] (degrees 15
// and 16: the first omitted terms are 5e-17 and 2e-18).  Coefficients are in
// constant memory, which the FP64 instructions read as operands.  Free of
// branches, so that the entries of a thread interleave; larger arguments go to
// the library (sincos_any), tested once per step.
constexpr int kReduceMax = 0x40f86a00;   // high word of 1e5
__constant__ double kSin[7] = {-1.0 / 1307674368000.0, 1.0 / 6227020800.0, -1.0 / 39916800.0, 1.0 / 362880.0,
                               -1.0 / 5040.0, 1.0 / 120.0, -1.0 / 6.0};   // 1/15!, 1/13!, ..., 1/3!
__constant__ double kCos[7] = {1.0 / 20922789888000.0, -1.0 / 87178291200.0, 1.0 / 479001600.0, -1.0 / 3628800.0,
                               1.0 / 40320.0, -1.0 / 720.0, 1.0 / 24.0};  // 1/16!, 1/14!, ..., 1/4!
__constant__ double kRed[4] = {0.63661977236758134308, 6755399441055744.0,   // 2/pi, 1.5 * 2^52
                               1.57079632679489661923, 6.12323399573676588613e-17};   // pi/2 in two parts

__device__ __noinline__ double2 sincos_any(double x)
{
    double2 v;
    sincos(x, &v.x, &v.y);
    return v;
}

__device__ __forceinline__ void sincos64(double x, double &s, double &c)
{
    const double t = fma(x, kRed[0], kRed[1]);
    const int n = __double2loint(t);
    const double q = t - kRed[1];
    const double d = fma(-q, kRed[3], fma(-q, kRed[2], x));
    const double d2 = d * d;
    double ps = kSin[0], pc = kCos[0];
    #pragma unroll
    for (int k = 1; k < 7; ++k)
    {
        ps = fma(ps, d2, kSin[k]);
        pc = fma(pc, d2, kCos[k]);
    }
    const double sd = fma(d * d2, ps, d);
    const double cd = fma(fma(pc, d2, -0.5), d2, 1.0);
    // x = n pi/2 + d
    const double a = (n & 1) ? cd : sd, b = (n & 1) ? sd : cd;
    s = __hiloint2double(__double2hiint(a) ^ ((n & 2) << 30), __double2loint(a));
    c = __hiloint2double(__double2hiint(b) ^ (((n + 1) & 2) << 30), __double2loint(b));
}

// 1 / sqrt(x): the hardware's approximation y (about 20 bits) and one step of
// third order of Householder's method (A. S. Householder, The Numerical Treatment
// of a Single Nonlinear Equation, 1970), which for y^-2 = x is the binomial series
// of (1 - e)^(-1/2) up to e^2: y (1 + e/2 + 3 e^2/8) with e = 1 - x y^2.
__device__ __forceinline__ double rsqrt64(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y * y, 1.0);
    return fma(y * e, fma(e, 0.375, 0.5), y);
}

__device__ __forceinline__ void dmma(double (&c)[4], const double (&a)[4], double2 b)
{
    asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b.x), "d"(b.y));
}

// sin, cos and 1 / sqrt(|x|) of each x as the kernels below evaluate them, then CUDA's
__global__ void math_probe_kernel(int64_t n, const double *__restrict__ x, double *__restrict__ out)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s, c;
    sincos64(x[i], s, c);
    const double2 v = sincos_any(x[i]);
    const bool large = (__double2hiint(x[i]) & 0x7fffffff) >= kReduceMax;
    out[i] = large ? v.x : s;
    out[n + i] = large ? v.y : c;
    out[2 * n + i] = rsqrt64(fabs(x[i]));
    out[3 * n + i] = v.x;
    out[4 * n + i] = v.y;
    out[5 * n + i] = rsqrt(fabs(x[i]));
}

struct Args
{
    const double *pts4, *tnrm4;   // targets, their normals (adjoint double layer only)
    int m, self, off;             // self: target i is source off + i and that pair is excluded
    const double *src4, *nrm4;    // sources and their normals
    const double2 *B;             // n x wc
    double2 *out;                 // splits x m x wc
    const ChunkParamsD *prm;
    int n, wc, wcs, cols, per_split;   // cols: real columns per set
};

// Entry evaluators.  Target: what a thread keeps per target.  pair(): what the
// wavenumbers of a unit share; entry(): one kernel entry.
template <bool SL, bool DL, bool ADL, bool RI>
struct BoundaryEntry
{
    static constexpr bool kSourceNormal = DL;
    struct Target { double x[3], nu[ADL ? 3 : 1]; };
    struct Pair { double ri, r, dmu, dnu; };
    static __device__ __forceinline__ void load(Target &t, const Args &a, int i)
    {
        #pragma unroll
        for (int q = 0; q < 3; ++q) t.x[q] = i < a.m ? a.pts4[4 * (int64_t)i + q] : 0.0;
        if (ADL)
        {
            #pragma unroll
            for (int q = 0; q < 3; ++q) t.nu[ADL ? q : 0] = i < a.m ? a.tnrm4[4 * (int64_t)i + q] : 0.0;
        }
    }
    static __device__ __forceinline__ Pair pair(const Target &t, const double (&y)[3], const double (&mu)[3], bool skip)
    {
        Pair p;
        const double zx = y[0] - t.x[0], zy = y[1] - t.x[1], zz = y[2] - t.x[2];
        const double r2 = fma(zz, zz, fma(zy, zy, zx * zx));
        const double ri = rsqrt64(r2);
        p.ri = skip ? 0.0 : ri;
        p.r = r2 * p.ri;
        p.dmu = p.dnu = 0.0;
        if (DL || ADL)
        {
            const double ri3 = p.ri * p.ri * p.ri;
            if (DL) p.dmu = fma(zz, mu[2], fma(zy, mu[1], zx * mu[0])) * ri3;
            if (ADL) p.dnu = fma(zz, t.nu[ADL ? 2 : 0], fma(zy, t.nu[ADL ? 1 : 0], zx * t.nu[0])) * ri3;
        }
        return p;
    }
    // q: kappa, c1, -c2, c3.  A = e^{i k r} h,  h = c1 / r + u - i k r u,  u = -(c2 dmu - c3 dnu)
    static __device__ __forceinline__ double phase(const Pair &p, const double *q) { return q[0] * p.r; }
    static __device__ __forceinline__ void entry(const Pair &p, const double *q, double kr, double sn, double cs,
                                                 double &ar, double &ai)
    {
        double ux = 0.0, uy = 0.0;
        if (DL) ux = q[3] * p.dmu;
        if (ADL) ux = fma(q[5], p.dnu, ux);
        if (!RI && DL) uy = q[4] * p.dmu;
        if (!RI && ADL) uy = fma(q[6], p.dnu, uy);
        double hx = ux, hy = 0.0;
        if (SL) hy = q[2] * p.ri;
        if (DL || ADL) hy = fma(-kr, ux, hy);
        if (!RI)
        {
            if (SL) hx = fma(q[1], p.ri, hx);
            if (DL || ADL)
            {
                hx = fma(kr, uy, hx);
                hy += uy;
            }
        }
        ar = fma(-hy, sn, hx * cs);
        ai = fma(hy, cs, hx * sn);
    }
};

template <bool SL, bool DL>
struct FarEntry
{
    static constexpr bool kSourceNormal = DL;
    struct Target { double x[3]; };
    struct Pair { double xy, xmu; };
    static __device__ __forceinline__ void load(Target &t, const Args &a, int i)
    {
        #pragma unroll
        for (int q = 0; q < 3; ++q) t.x[q] = i < a.m ? a.pts4[4 * (int64_t)i + q] : 0.0;
    }
    static __device__ __forceinline__ Pair pair(const Target &t, const double (&y)[3], const double (&mu)[3], bool)
    {
        Pair p;   // a source past the end has a zero right-hand side and a finite entry
        p.xy = fma(y[2], t.x[2], fma(y[1], t.x[1], y[0] * t.x[0]));
        p.xmu = DL ? fma(mu[2], t.x[2], fma(mu[1], t.x[1], mu[0] * t.x[0])) : 0.0;
        return p;
    }
    static __device__ __forceinline__ double phase(const Pair &p, const double *q) { return q[0] * p.xy; }
    static __device__ __forceinline__ void entry(const Pair &p, const double *q, double, double sn, double cs,
                                                 double &ar, double &ai)
    {
        double fx = SL ? q[1] : 0.0, fy = SL ? q[2] : 0.0;   // c1 - i k c2 (x.mu)
        if (DL)
        {
            const double dk = q[0] * p.xmu;
            fx = fma(-q[4], dk, fx);   // q[3], q[4] = -c2
            fy = fma(q[3], dk, fy);
        }
        ar = fma(fy, sn, fx * cs);
        ai = fma(fy, cs, -fx * sn);
    }
};

// E wavenumbers of NT * 8 columns each
template <int E, int NT>
struct Smem
{
    double2 frag[kStage / 8][E * NT][2][32];   // per step, 8 columns and part (re, im): the B registers of each lane
    double tot[E * NT * 8][kThreads];          // running totals, private to the thread
    double geo[kStage][6];                     // source position, normal
    double prm[E][8];                          // kappa, c1, -c2, c3
};

template <class Entry, int E, int NT>
__global__ void __launch_bounds__(kThreads, 2) d64_kernel(const Args a)
{
    chain_wait();
    extern __shared__ __align__(16) uint8_t raw[];
    Smem<E, NT> &sm = *reinterpret_cast<Smem<E, NT> *>(raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int col0 = blockIdx.y * E * a.cols;
    const int jb = blockIdx.z * a.per_split, je = min(a.n, jb + a.per_split);
    const int i0 = (blockIdx.x * 4 + warp) * kWarpTargets + g, i1 = i0 + 8;
    const int self0 = a.self ? a.off + i0 : -1, self1 = a.self ? a.off + i1 : -1;
    typename Entry::Target x0, x1;
    Entry::load(x0, a, i0);
    Entry::load(x1, a, i1);
    if (tid < E)
    {
        const ChunkParamsD &q = a.prm[col0 / a.wcs + tid];
        double *p = sm.prm[tid];
        p[0] = q.kappa;
        p[1] = q.c[1].x; p[2] = q.c[1].y;
        p[3] = -q.c[2].x; p[4] = -q.c[2].y;
        p[5] = q.c[3].x; p[6] = q.c[3].y;
    }
    #pragma unroll
    for (int q = 0; q < E * NT * 8; ++q) sm.tot[q][tid] = 0.0;
    double acc[E * NT][2][4];
    #pragma unroll
    for (int q = 0; q < E * NT; ++q)
        #pragma unroll
        for (int v = 0; v < 4; ++v) acc[q][0][v] = acc[q][1][v] = 0.0;
    auto flush = [&]() {
        #pragma unroll
        for (int q = 0; q < E * NT; ++q)
            #pragma unroll
            for (int v = 0; v < 4; ++v)
            {
                sm.tot[q * 8 + 2 * v][tid] += acc[q][0][v];
                sm.tot[q * 8 + 2 * v + 1][tid] += acc[q][1][v];
                acc[q][0][v] = acc[q][1][v] = 0.0;
            }
    };
    int in_segment = 0;
    for (int j0 = jb; j0 < je; j0 += kStage)
    {
        __syncthreads();
        // One B register pair per turn: sources 8 k + t' and 8 k + 4 + t', column 8 q + g'; the
        // loads of all turns are in flight together, the stores are 16 bytes per lane in lane order.
        constexpr int kTurns = kStage / 8 * E * NT * 32 / kThreads;
        double2 b0[kTurns], b1[kTurns];
        #pragma unroll
        for (int e = 0; e < kTurns; ++e)
        {
            const int kq = e * 4 + warp, j = j0 + kq / (E * NT) * 8 + t;
            const int set = kq % (E * NT) / NT, c = kq % NT * 8 + g;   // column of the set
            const double2 *src = a.B + (int64_t)j * a.wc + col0 + set * a.cols + c;
            b0[e] = j < je && c < a.cols ? *src : make_double2(0.0, 0.0);
            b1[e] = j + 4 < je && c < a.cols ? src[4 * (int64_t)a.wc] : make_double2(0.0, 0.0);
        }
        #pragma unroll
        for (int e = 0; e < kTurns; ++e)
        {
            const int kq = e * 4 + warp;
            double2(*f)[32] = sm.frag[kq / (E * NT)][kq % (E * NT)];
            f[0][lane] = make_double2(b0[e].x, b1[e].x);
            f[1][lane] = make_double2(b0[e].y, b1[e].y);
        }
        for (int e = tid; e < kStage * 3; e += kThreads)
        {
            const int s = e / 3, q = e - 3 * s, j = j0 + s;
            sm.geo[s][q] = j < je ? a.src4[4 * (int64_t)j + q] : 0.0;
            if (Entry::kSourceNormal) sm.geo[s][3 + q] = j < je ? a.nrm4[4 * (int64_t)j + q] : 0.0;
        }
        __syncthreads();
        const int steps = min(kStage, je - j0 + 7) >> 3;
        #pragma unroll 1
        for (int k = 0; k < steps; ++k)
        {
            typename Entry::Pair p[4];   // (i0, t), (i1, t), (i0, t + 4), (i1, t + 4)
            #pragma unroll
            for (int h = 0; h < 2; ++h)
            {
                const int s = 8 * k + 4 * h + t, j = j0 + s;
                const double2 *gs = reinterpret_cast<const double2 *>(sm.geo[s]);
                const double2 ga = gs[0], gb = gs[1];
                const double2 gc = Entry::kSourceNormal ? gs[2] : make_double2(0.0, 0.0);
                const double y[3] = {ga.x, ga.y, gb.x}, mu[3] = {gb.y, gc.x, gc.y};
                p[2 * h] = Entry::pair(x0, y, mu, j == self0 || j >= je);
                p[2 * h + 1] = Entry::pair(x1, y, mu, j == self1 || j >= je);
            }
            #pragma unroll
            for (int e = 0; e < E; ++e)
            {
                double th[4], sn[4], cs[4], ar[4], ai[4], nai[4];
                bool large = false;
                #pragma unroll
                for (int v = 0; v < 4; ++v)
                {
                    th[v] = Entry::phase(p[v], sm.prm[e]);
                    sincos64(th[v], sn[v], cs[v]);
                    large |= (__double2hiint(th[v]) & 0x7fffffff) >= kReduceMax;
                }
                if (large)
                {
                    #pragma unroll
                    for (int v = 0; v < 4; ++v)
                    {
                        const double2 sc = sincos_any(th[v]);
                        sn[v] = sc.x;
                        cs[v] = sc.y;
                    }
                }
                #pragma unroll
                for (int v = 0; v < 4; ++v)
                {
                    Entry::entry(p[v], sm.prm[e], th[v], sn[v], cs[v], ar[v], ai[v]);
                    nai[v] = __hiloint2double(__double2hiint(ai[v]) ^ 0x80000000, __double2loint(ai[v]));
                }
                #pragma unroll
                for (int q = 0; q < NT; ++q)
                {
                    const double2(*f)[32] = sm.frag[k][e * NT + q];
                    const double2 br = f[0][lane], bi = f[1][lane];
                    dmma(acc[e * NT + q][0], ar, br);
                    dmma(acc[e * NT + q][1], ar, bi);
                    dmma(acc[e * NT + q][0], nai, bi);
                    dmma(acc[e * NT + q][1], ai, br);
                }
            }
        }
        in_segment += kStage;
        if (in_segment >= kSegment)
        {
            flush();
            in_segment = 0;
        }
    }
    flush();
    chain_next();
    // accumulator v of tile q: row g + 8 (v / 2), column 8 q + 2 t + v % 2; with a cluster
    // of S parts, block r adds accumulators r, r + S, ... of all of them in order
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    if (S > 1) cluster.sync();
    double2 *out = a.out + (int64_t)(blockIdx.z / S) * a.m * a.wc + col0;
    for (int e = rank; e < E * NT * 4; e += S)
    {
        const int q = e / 4, v = e % 4;
        double2 o = make_double2(0.0, 0.0);
        for (int s = 0; s < S; ++s)
        {
            const double *tot = S > 1 ? cluster.map_shared_rank(&sm.tot[2 * e][tid], s) : &sm.tot[2 * e][tid];
            o.x += tot[0];
            o.y += tot[kThreads];
        }
        const int i = v < 2 ? i0 : i1, c = q % NT * 8 + 2 * t + (v & 1);
        if (i < a.m && c < a.cols) out[(int64_t)i * a.wc + q / NT * a.cols + c] = o;
    }
    if (S > 1) cluster.sync();   // no block leaves while its totals are read
}

template <class Entry, int E, int NT>
void launch(const Args &a, dim3 grid, int cluster, cudaStream_t st)
{
    constexpr size_t bytes = sizeof(Smem<E, NT>);
    // the shared-memory limit is a per-device attribute of the function
    int dev = 0;
    BAEMM_CUDA(cudaGetDevice(&dev));
    static std::mutex mu;
    static bool done[64] = {};
    {
        std::lock_guard<std::mutex> lock(mu);
        if (dev < 0 || dev >= 64 || !done[dev])
        {
            BAEMM_CUDA(cudaFuncSetAttribute(d64_kernel<Entry, E, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)bytes));
            if (dev >= 0 && dev < 64) done[dev] = true;
        }
    }
    launch_chained(d64_kernel<Entry, E, NT>, grid, kThreads, bytes, st, cluster, a);
}

template <class Entry>
void by_unit(const D64Unit &u, const Args &a, dim3 grid, int cluster, cudaStream_t st)
{
    if (u.sets == 2 && u.tiles == 2) launch<Entry, 2, 2>(a, grid, cluster, st);
    else if (u.sets == 2) launch<Entry, 2, 1>(a, grid, cluster, st);
    else if (u.tiles == 4) launch<Entry, 1, 4>(a, grid, cluster, st);
    else if (u.tiles == 2) launch<Entry, 1, 2>(a, grid, cluster, st);
    else launch<Entry, 1, 1>(a, grid, cluster, st);
}

template <bool RI>
void by_layers(int code, const D64Unit &u, const Args &a, dim3 grid, int cluster, cudaStream_t st)
{
    switch (code)
    {
        case 1: by_unit<BoundaryEntry<true, false, false, RI>>(u, a, grid, cluster, st); break;
        case 2: by_unit<BoundaryEntry<false, true, false, RI>>(u, a, grid, cluster, st); break;
        case 3: by_unit<BoundaryEntry<true, true, false, RI>>(u, a, grid, cluster, st); break;
        case 4: by_unit<BoundaryEntry<false, false, true, RI>>(u, a, grid, cluster, st); break;
        case 5: by_unit<BoundaryEntry<true, false, true, RI>>(u, a, grid, cluster, st); break;
        case 6: by_unit<BoundaryEntry<false, true, true, RI>>(u, a, grid, cluster, st); break;
        case 7: by_unit<BoundaryEntry<true, true, true, RI>>(u, a, grid, cluster, st); break;
        default: break;
    }
}

dim3 grid_of(const D64Unit &u, int64_t m, int wc, SourceSplit split)
{
    return dim3(ceil_div(m, 4 * kWarpTargets), wc / u.columns(), split.parts());
}

// sources per part, whole steps of 8
int part_of(int64_t n, SourceSplit split) { return ceil_div(ceil_div(n, split.parts()), 8) * 8; }

} // namespace

D64Unit d64_unit(int wc, int wcs)
{
    D64Unit u;
    u.tiles = wcs >= 32 ? 4 : wcs >= 16 ? 2 : 1;
    u.cols = std::min(wcs, u.tiles * 8);
    u.sets = wcs <= 16 && (wc / wcs) % 2 == 0 ? 2 : 1;
    return u;
}

int64_t d64_ctas(const D64Unit &u, int64_t m, int wc) { return (int64_t)ceil_div(m, 4 * kWarpTargets) * (wc / u.columns()); }

void d64_math_probe(int64_t n, const double *x, double *out)
{
    DevBuf<double> dx, dy;
    BAEMM_CUDA(cudaMemcpy(dx.reserve(n), x, n * sizeof(double), cudaMemcpyHostToDevice));
    math_probe_kernel<<<ceil_div(n, 256), 256>>>(n, dx.p, dy.reserve(6 * n));
    BAEMM_LAUNCH_CHECK();
    BAEMM_CUDA(cudaMemcpy(out, dy.p, 6 * n * sizeof(double), cudaMemcpyDeviceToHost));
}

void launch_boundary_d64(const MeshDev &m, const OpFlags &f, const ChunkParamsD *prm, int wc, int wcs,
                         const DenseTargets<double> &tg, const double2 *Btri, double2 *out, SourceSplit split,
                         cudaStream_t st)
{
    const D64Unit u = d64_unit(wc, wcs);
    const Args a{tg.pts4, m.nrm_d + 4 * (int64_t)tg.off, tg.m, tg.self, tg.off, m.mid_d, m.nrm_d, Btri, out, prm,
                 (int)m.nt, wc, wcs, u.cols, part_of(m.nt, split)};
    const dim3 grid = grid_of(u, tg.m, wc, split);
    const int cluster = split.cluster;
    const int code = (f.sl() ? 1 : 0) | (f.dl() ? 2 : 0) | (f.adl() ? 4 : 0);
    if (!f.re_sl_d && !f.im_dl_d && !f.im_adl_d) by_layers<true>(code, u, a, grid, cluster, st);
    else by_layers<false>(code, u, a, grid, cluster, st);
    BAEMM_LAUNCH_CHECK();
}

void launch_farfield_d64(const MeshDev &m, const OpFlags &f, const ChunkParamsD *prm, int wc, int wcs,
                         const double2 *Btri, double2 *partial, SourceSplit split, cudaStream_t st)
{
    const D64Unit u = d64_unit(wc, wcs);
    const Args a{m.meas_d, nullptr, (int)m.nm, 0, 0, m.mid_d, m.nrm_d, Btri, partial, prm,
                 (int)m.nt, wc, wcs, u.cols, part_of(m.nt, split)};
    const dim3 grid = grid_of(u, m.nm, wc, split);
    const int cluster = split.cluster;
    if (f.sl() && f.dl()) by_unit<FarEntry<true, true>>(u, a, grid, cluster, st);
    else if (f.sl()) by_unit<FarEntry<true, false>>(u, a, grid, cluster, st);
    else by_unit<FarEntry<false, true>>(u, a, grid, cluster, st);
    BAEMM_LAUNCH_CHECK();
}

} // namespace baemm
