// Integer topology of a mesh on the device: AvOp columns sorted per triangle
// (Initialize.hpp:307-313), AvOp^T as a vertex -> triangle CSR in ascending
// triangle order (Initialize.hpp:315) and the sparsity pattern of the P1 mass
// matrix (Initialize.hpp:329-334).  Rows are filled through atomic counters and
// sorted afterwards, so the result does not depend on timing.
//
// Bound by launches and latency: six small kernels (ten where the vertices take
// more than one tile of the scan) and one host round trip.  Setting a mesh (its copies and geometry included) takes 0.22 ms
// with 5120 triangles, 0.28 with 41666, 0.65 with 153600; with the topology built
// on the host (a sort of 9 nt 64-bit keys) 1.9, 25.8 and 111 ms.
#include "ops.cuh"

#include <algorithm>

namespace baemm
{
namespace
{

constexpr int kScanThreads = 256, kScanItems = 8, kScanTile = kScanThreads * kScanItems;

__global__ void count_kernel(int64_t nt, const int32_t *__restrict__ tris, int32_t *__restrict__ sorted,
                             int32_t *__restrict__ count)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt) return;
    const int32_t a = tris[3 * t], b = tris[3 * t + 1], c = tris[3 * t + 2];
    sorted[3 * t] = min(a, min(b, c));
    sorted[3 * t + 1] = max(min(a, b), min(max(a, b), c));
    sorted[3 * t + 2] = max(a, max(b, c));
    atomicAdd(&count[a], 1);
    atomicAdd(&count[b], 1);
    atomicAdd(&count[c], 1);
}

// out = exclusive sums of in within a tile, total[tile] = the tile's sum; *most >= every item
__global__ void __launch_bounds__(kScanThreads)
scan_tiles_kernel(int64_t n, const int32_t *__restrict__ in, int32_t *__restrict__ out, int32_t *__restrict__ total,
                  int32_t *__restrict__ most)
{
    __shared__ int32_t warp_sum[kScanThreads / 32];
    const int64_t i0 = (int64_t)blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    int32_t v[kScanItems], sum = 0, top = 0;
    #pragma unroll
    for (int q = 0; q < kScanItems; ++q)
    {
        v[q] = i0 + q < n ? in[i0 + q] : 0;
        sum += v[q];
        top = max(top, v[q]);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t inc = sum;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int32_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) warp_sum[warp] = inc;
    __syncthreads();
    int32_t before = inc - sum;
    for (int w = 0; w < warp; ++w) before += warp_sum[w];
    #pragma unroll
    for (int q = 0; q < kScanItems; ++q)
    {
        if (i0 + q < n) out[i0 + q] = before;
        before += v[q];
    }
    if (threadIdx.x == kScanThreads - 1) total[blockIdx.x] = before;
    if (most)
    {
        top = __reduce_max_sync(0xffffffffu, top);
        if (lane == 0) atomicMax(most, top);
    }
}

// exclusive sums of the tile totals in place, one block
__global__ void __launch_bounds__(1024) scan_totals_kernel(int tiles, int32_t *total)
{
    __shared__ int32_t warp_sum[32];
    __shared__ int32_t carry;
    if (threadIdx.x == 0) carry = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int b = 0; b < tiles; b += 1024)
    {
        const int i = b + threadIdx.x;
        const int32_t v = i < tiles ? total[i] : 0;
        int32_t inc = v;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int32_t u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (lane == 31) warp_sum[warp] = inc;
        __syncthreads();
        int32_t before = carry + inc - v;
        for (int w = 0; w < warp; ++w) before += warp_sum[w];
        if (i < tiles) total[i] = before;
        __syncthreads();   // carry has been read
        if (threadIdx.x == 1023) carry = before + v;
        __syncthreads();
    }
}

__global__ void scan_add_kernel(int64_t n, const int32_t *__restrict__ total, int32_t *__restrict__ out)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] += total[i / kScanTile];
}

__global__ void fill_kernel(int64_t nt, const int32_t *__restrict__ tris, const int32_t *__restrict__ outer,
                            int32_t *__restrict__ cursor, int32_t *__restrict__ inner)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt) return;
    #pragma unroll
    for (int q = 0; q < 3; ++q)
    {
        const int32_t v = tris[3 * t + q];
        inner[outer[v] + atomicAdd(&cursor[v], 1)] = (int32_t)t;
    }
}

// Sorts the vertex's triangles and lists the vertices of those triangles, each
// once, ascending, in its slots (2 degree + 1 of them); nothing where a vertex
// has more than kTopologyDegree triangles (the insertion sorts are quadratic).
__global__ void rows_kernel(int64_t nv, const int32_t *__restrict__ tris, const int32_t *__restrict__ outer,
                            const int32_t *__restrict__ most, int32_t *inner, int32_t *slots, int32_t *__restrict__ count)
{
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v > nv) return;
    if (v == nv || *most > kTopologyDegree)
    {
        count[v] = 0;
        return;
    }
    const int32_t e0 = outer[v], e1 = outer[v + 1];
    for (int32_t e = e0 + 1; e < e1; ++e)
    {
        const int32_t t = inner[e];
        int32_t i = e;
        for (; i > e0 && inner[i - 1] > t; --i) inner[i] = inner[i - 1];
        inner[i] = t;
    }
    int32_t *s = slots + v + 2 * (int64_t)e0, n = 0;
    for (int32_t e = e0; e < e1; ++e)
        for (int q = 0; q < 3; ++q)
        {
            const int32_t w = tris[3 * (int64_t)inner[e] + q];
            int32_t i = n;
            while (i > 0 && s[i - 1] > w) --i;
            if (i > 0 && s[i - 1] == w) continue;
            for (int32_t j = n; j > i; --j) s[j] = s[j - 1];
            s[i] = w;
            ++n;
        }
    count[v] = n;
}

__global__ void pack_kernel(int64_t nv, const int32_t *__restrict__ avt_outer, const int32_t *__restrict__ slots,
                            const int32_t *__restrict__ outer, int32_t *__restrict__ inner)
{
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nv) return;
    const int32_t *s = slots + v + 2 * (int64_t)avt_outer[v];
    const int32_t e0 = outer[v], n = outer[v + 1] - e0;
    for (int32_t j = 0; j < n; ++j) inner[e0 + j] = s[j];
}

void scan(int64_t n, const int32_t *in, int32_t *out, int32_t *total, int32_t *most, cudaStream_t st)
{
    const int tiles = ceil_div(n, kScanTile);
    scan_tiles_kernel<<<tiles, kScanThreads, 0, st>>>(n, in, out, total, most);
    BAEMM_LAUNCH_CHECK();
    if (tiles == 1) return;
    scan_totals_kernel<<<1, 1024, 0, st>>>(tiles, total);
    BAEMM_LAUNCH_CHECK();
    scan_add_kernel<<<ceil_div(n, 256), 256, 0, st>>>(n, total, out);
    BAEMM_LAUNCH_CHECK();
}

} // namespace

int64_t launch_topology(MeshDev &m, DevBuf<int32_t> &scratch, int32_t *host2, cudaStream_t st)
{
    const int64_t nv = m.nv, nt = m.nt, tiles = ceil_div(nv + 1, kScanTile);
    m.tri_sorted.reserve(3 * nt);
    m.avt_outer.reserve(nv + 1);
    m.avt_inner.reserve(3 * nt);
    m.mass_outer.reserve(nv + 1);
    // scratch: counts (then cursors), most | counts of the mass rows | totals | slots
    int32_t *count = scratch.reserve(2 * (nv + 1) + 1 + tiles + nv + 6 * nt);
    int32_t *most = count + nv + 1, *rows = most + 1, *total = rows + nv + 1, *slots = total + tiles;
    const int T = 128;
    BAEMM_CUDA(cudaMemsetAsync(count, 0, (nv + 2) * sizeof(int32_t), st));
    count_kernel<<<ceil_div(nt, T), T, 0, st>>>(nt, m.tris, m.tri_sorted, count);
    BAEMM_LAUNCH_CHECK();
    scan(nv + 1, count, m.avt_outer, total, most, st);
    BAEMM_CUDA(cudaMemsetAsync(count, 0, nv * sizeof(int32_t), st));
    fill_kernel<<<ceil_div(nt, T), T, 0, st>>>(nt, m.tris, m.avt_outer, count, m.avt_inner);
    BAEMM_LAUNCH_CHECK();
    rows_kernel<<<ceil_div(nv + 1, T), T, 0, st>>>(nv, m.tris, m.avt_outer, most, m.avt_inner, slots, rows);
    BAEMM_LAUNCH_CHECK();
    scan(nv + 1, rows, m.mass_outer, total, nullptr, st);
    BAEMM_CUDA(cudaMemcpyAsync(&host2[0], most, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    BAEMM_CUDA(cudaMemcpyAsync(&host2[1], m.mass_outer + nv, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    wait_stream(st);
    if (host2[0] > kTopologyDegree) return -1;
    m.mass_inner.reserve(std::max(host2[1], 1));
    pack_kernel<<<ceil_div(nv, T), T, 0, st>>>(nv, m.avt_outer, slots, m.mass_outer, m.mass_inner);
    BAEMM_LAUNCH_CHECK();
    return host2[1];
}

} // namespace baemm
