/*
 * ag_bins.cu -- device planner of the solve kernel's bins (ag_bins.h).
 *
 * Rows are cut into bins by a scan of their weights: row v belongs to bin
 * floor(W(v) / quantum) + (its graph of a union), W the weight before it, so
 * every bin's first row is one binary search and no walk over the rows is
 * needed.  One CTA per bin then sorts the bin's rows by length with a
 * shared-memory histogram and writes the lists.
 */
#include <cub/cub.cuh>
#include <string.h>

#include "ag_bins.h"

#define AG_BINS_BLK 256
#define AG_BINS_W40 ((1ull << 40) - 1ull)

__global__ void ag_bins_weight_kernel(const uint32_t *off, uint32_t n, uint64_t *w)
{
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += (uint64_t)gridDim.x * blockDim.x) {
        if (v == n) {
            w[n] = 0;
            continue;
        }
        const uint32_t d = off[v + 1] - off[v];
        uint64_t x = 1;
        if (d > AG_BIN_HUB)
            x += (uint64_t)((d - 1u) / AG_BIN_HUB + 1u) << 40;
        else
            x += d > AG_BIN_SEQ ? (d + 3u) & ~3u : d;
        w[v] = x;
    }
}

/* index of the graph holding row r */
__device__ __forceinline__ uint32_t ag_bins_graph(const uint32_t *gstart, uint32_t ngraphs, uint32_t r)
{
    uint32_t lo = 0, hi = ngraphs;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (gstart[mid] <= r)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

struct AgBinsArgs
{
    const uint32_t *off, *gstart;
    const uint64_t *pre;
    uint32_t n, ngraphs, quantum, nbins;
    AgBin *bins;
    uint4 *hubs;
    uint32_t *brow, *ubase;
    uint64_t hub_slots;
};

/* the first row of bin k (n when no later row exists) */
__device__ __forceinline__ uint32_t ag_bins_first(const AgBinsArgs &a, uint32_t k)
{
    uint32_t lo = 0, hi = a.n;
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        const uint32_t g = a.gstart ? ag_bins_graph(a.gstart, a.ngraphs, mid) : 0u;
        if ((uint32_t)((a.pre[mid] & AG_BINS_W40) / a.quantum) + g < k)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

/* lengths to sort keys, longest first: 48 classes of long rows (eight per
 * power of two), then short rows by exact length */
#define AG_BINS_KEYS (48u + AG_BIN_SEQ)
__device__ __forceinline__ uint32_t ag_bins_key(uint32_t d)
{
    if (d <= AG_BIN_SEQ)
        return 48u + AG_BIN_SEQ - d;
    const uint32_t oct = 31u - __clz(d - 1u);
    return 47u - ((oct - 5u) * 8u + (((d - 1u) >> (oct - 3u)) & 7u));
}

__global__ void __launch_bounds__(AG_BINS_BLK) ag_bins_rows_kernel(const AgBinsArgs a)
{
    __shared__ uint32_t hist[AG_BINS_KEYS];
    __shared__ uint32_t s_r0, s_r1, s_nlong, s_nshort, s_total;
    extern __shared__ uint32_t list[]; /* quantum + 64 entries, then the units' sizes */
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, bin = blockIdx.x;
    if (tid < 2)
        (tid ? s_r1 : s_r0) = ag_bins_first(a, bin + tid);
    for (uint32_t i = tid; i < AG_BINS_KEYS; i += AG_BINS_BLK)
        hist[i] = 0;
    __syncthreads();
    const uint32_t r0 = s_r0, nrows = s_r1 - r0;
    for (uint32_t i = tid; i < nrows; i += AG_BINS_BLK) {
        const uint32_t d = a.off[r0 + i + 1] - a.off[r0 + i];
        if (d && d <= AG_BIN_HUB)
            atomicAdd(&hist[ag_bins_key(d)], 1u);
    }
    __syncthreads();
    if (tid == 0) {
        uint32_t p = 0, nl = 0;
        for (uint32_t k = 0; k < AG_BINS_KEYS; ++k) {
            if (k == 48) {
                nl = p;
                p = (p + 31u) & ~31u; /* short rows start a unit */
            }
            const uint32_t c = hist[k];
            hist[k] = p;
            p += c;
        }
        s_nlong = nl;
        s_nshort = p - ((nl + 31u) & ~31u);
    }
    __syncthreads();
    const uint32_t ulong = (s_nlong + 31u) >> 5, units = ulong + ((s_nshort + 31u) >> 5);
    uint32_t *usz = list + 32u * units;
    for (uint32_t i = tid; i < 32u * units; i += AG_BINS_BLK)
        list[i] = 0;
    __syncthreads();
    for (uint32_t i = tid; i < nrows; i += AG_BINS_BLK) {
        const uint32_t d = a.off[r0 + i + 1] - a.off[r0 + i];
        if (d && d <= AG_BIN_HUB)
            list[atomicAdd(&hist[ag_bins_key(d)], 1u)] = i | (d << 16);
    }
    __syncthreads();
    for (uint32_t u = warp; u < units; u += AG_BINS_BLK / 32) {
        const uint32_t len = list[32u * u + lane] >> 16;
        const uint32_t sz = u < ulong ? __reduce_add_sync(0xffffffffu, (len + 3u) & ~3u)
                                      : 32u * __reduce_max_sync(0xffffffffu, len);
        if (lane == 0)
            usz[u] = sz;
    }
    __syncthreads();
    if (warp == 0) {
        uint32_t run = 0;
        for (uint32_t u0 = 0; u0 < units; u0 += 32) {
            const uint32_t x = u0 + lane < units ? usz[u0 + lane] : 0u;
            uint32_t inc = x;
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o)
                    inc += t;
            }
            if (u0 + lane < units)
                usz[u0 + lane] = run + inc - x;
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0)
            s_total = run;
    }
    __syncthreads();
    const uint32_t lb = ag_bin_list(r0, bin);
    for (uint32_t i = tid; i < 32u * units; i += AG_BINS_BLK)
        a.brow[lb + i] = list[i];
    for (uint32_t u = tid; u < units; u += AG_BINS_BLK)
        a.ubase[(lb >> 5) + u] = usz[u];
    if (tid == 0) {
        AgBin b;
        b.r0 = r0;
        b.nrows = nrows;
        b.nlong = s_nlong;
        b.nshort = s_nshort;
        b.nslots = s_total;
        b.gid = a.gstart && nrows ? ag_bins_graph(a.gstart, a.ngraphs, r0) : 0u;
        /* slots of the bins before it, at most */
        b.sbase = a.hub_slots + (((a.pre[r0] & AG_BINS_W40) + 3ull) & ~3ull) + (uint64_t)bin * (AG_BIN_PAD + 64u);
        a.bins[bin] = b;
    }
}

__global__ void ag_bins_hubs_kernel(const AgBinsArgs a)
{
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < a.n; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t d = a.off[v + 1] - a.off[v];
        if (d <= AG_BIN_HUB)
            continue;
        const uint32_t nch = (d - 1u) / AG_BIN_HUB + 1u, first = (uint32_t)(a.pre[v] >> 40);
        for (uint32_t c = 0; c < nch; ++c)
            a.hubs[first + c] = make_uint4((uint32_t)v, c, first,
                                           (min(AG_BIN_HUB, d - c * AG_BIN_HUB) - 1u) | (nch << 11));
    }
}

/* T: ids or weights */
template <typename T>
__global__ void __launch_bounds__(AG_BINS_BLK) ag_bins_ids_kernel(const uint32_t *off, const T *ids,
                                                                  const AgBin *bins, const uint4 *hubs, uint32_t nhub,
                                                                  const uint32_t *brow, const uint32_t *ubase,
                                                                  T *out)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (blockIdx.x < nhub) {
        const uint4 h = hubs[blockIdx.x];
        const uint32_t len = (h.w & (AG_BIN_HUB - 1u)) + 1u;
        const T *src = ids + off[h.x] + (size_t)h.y * AG_BIN_HUB;
        T *dst = out + (size_t)blockIdx.x * AG_BIN_HUB;
        for (uint32_t i = tid; i < AG_BIN_HUB; i += AG_BINS_BLK)
            dst[i] = i < len ? src[i] : T(0);
        return;
    }
    const uint32_t k = blockIdx.x - nhub;
    const AgBin b = bins[k];
    const uint32_t lb = ag_bin_list(b.r0, k);
    const uint32_t ulong = (b.nlong + 31u) >> 5, units = ulong + ((b.nshort + 31u) >> 5);
    for (uint32_t u = warp; u < units; u += AG_BINS_BLK / 32) {
        const uint32_t e = brow[lb + 32u * u + lane], len = e >> 16;
        const uint32_t o = len ? off[b.r0 + (e & 0xffffu)] : 0u;
        T *dst = out + b.sbase + ubase[(lb >> 5) + u];
        if (u < ulong) {
            for (int l = 0; l < 32; ++l) {
                const uint32_t n = __shfl_sync(0xffffffffu, len, l), ob = __shfl_sync(0xffffffffu, o, l);
                for (uint32_t i = lane; i < ((n + 3u) & ~3u); i += 32)
                    dst[i] = i < n ? ids[ob + i] : T(0);
                dst += (n + 3u) & ~3u;
            }
        } else {
            const uint32_t most = __shfl_sync(0xffffffffu, len, 0); /* longest first */
#pragma unroll 4
            for (uint32_t i = 0; i < most; ++i)
                dst[32u * i + lane] = i < len ? ids[o + i] : T(0);
        }
    }
}

/* ------------------------------------------------------------- host side */
static unsigned bins_grid(uint64_t n)
{
    uint64_t g = (n + 255) / 256;
    if (g > ag_sm_grid(16))
        g = ag_sm_grid(16);
    return g ? (unsigned)g : 1u;
}

extern "C" cudaError_t ag_bins_count(const uint32_t *row_off, uint32_t n, AgBinPlan *b, uint64_t *total_host,
                                     cudaStream_t s)
{
    size_t tb = 0;
    cudaError_t e = cub::DeviceScan::ExclusiveSum(nullptr, tb, (const uint64_t *)nullptr, (uint64_t *)nullptr,
                                                  (int)n + 1, s);
    if (e == cudaSuccess)
        e = cudaMallocAsync((void **)&b->pre, ((size_t)n + 1) * 8, s);
    if (e == cudaSuccess)
        e = cudaMallocAsync(&b->tmp, tb ? tb : 16, s);
    if (e != cudaSuccess)
        return e;
    ag_bins_weight_kernel<<<bins_grid((uint64_t)n + 1), 256, 0, s>>>(row_off, n, b->pre);
    e = cub::DeviceScan::ExclusiveSum(b->tmp, tb, b->pre, b->pre, (int)n + 1, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(total_host, b->pre + n, 8, cudaMemcpyDeviceToHost, s);
    return e;
}

extern "C" void ag_bins_shape(AgBinPlan *b, uint64_t total, uint32_t quantum, uint32_t ngraphs)
{
    const uint64_t w = total & AG_BINS_W40;
    b->quantum = quantum;
    b->buf = AG_BIN_BUF(quantum);
    b->nhub = (uint32_t)(total >> 40);
    b->nbins = w ? (uint32_t)((w - 1) / quantum) + (ngraphs ? ngraphs : 1u) : 0u;
    b->nslots = (uint64_t)b->nhub * AG_BIN_HUB + w + (uint64_t)b->nbins * (AG_BIN_PAD + 64u) + 64u;
}

extern "C" size_t ag_bins_brow_words(const AgBinPlan *b, uint32_t n) { return (size_t)n + 96u * ((size_t)b->nbins + 1u); }

static AgBinsArgs bins_args(const uint32_t *row_off, uint32_t n, const uint32_t *gstart, uint32_t ngraphs,
                            const AgBinPlan *b)
{
    AgBinsArgs a;
    memset(&a, 0, sizeof(a));
    a.off = row_off;
    a.gstart = ngraphs ? gstart : nullptr;
    a.pre = b->pre;
    a.n = n;
    a.ngraphs = ngraphs;
    a.quantum = b->quantum;
    a.nbins = b->nbins;
    a.bins = b->bins;
    a.hubs = b->hubs;
    a.brow = b->brow;
    a.ubase = b->ubase;
    a.hub_slots = (uint64_t)b->nhub * AG_BIN_HUB;
    return a;
}

extern "C" cudaError_t ag_bins_rows(const uint32_t *row_off, uint32_t n, const uint32_t *gstart, uint32_t ngraphs,
                                    AgBinPlan *b, cudaStream_t s)
{
    const AgBinsArgs a = bins_args(row_off, n, gstart, ngraphs, b);
    if (b->nbins) {
        /* the list holds every row and the two padded units, then the unit sizes */
        const uint32_t entries = b->quantum + 1u + 64u;
        const size_t smem = (size_t)(entries + entries / 32u + 4u) * 4u;
        cudaError_t e = cudaFuncSetAttribute(ag_bins_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess)
            return e;
        ag_bins_rows_kernel<<<b->nbins, AG_BINS_BLK, smem, s>>>(a);
    }
    if (b->nhub)
        ag_bins_hubs_kernel<<<bins_grid(n), 256, 0, s>>>(a);
    return cudaGetLastError();
}

extern "C" cudaError_t ag_bins_ids(const uint32_t *row_off, const uint32_t *ids, const float *w, const AgBinPlan *b,
                                   cudaStream_t s)
{
    const uint32_t grid = b->nbins + b->nhub;
    if (grid) {
        ag_bins_ids_kernel<<<grid, AG_BINS_BLK, 0, s>>>(row_off, ids, b->bins, b->hubs, b->nhub, b->brow, b->ubase, b->ids);
        if (b->w)
            ag_bins_ids_kernel<<<grid, AG_BINS_BLK, 0, s>>>(row_off, w, b->bins, b->hubs, b->nhub, b->brow, b->ubase, b->w);
    }
    return cudaGetLastError();
}
