/*
 * ag_units.cu -- device planner of the solve kernel's units (ag_units.h).
 *
 * One CTA per window sorts its rows by their quads (a stable block radix
 * sort), so that rows of equal size keep their order and a unit's rows lie
 * close together: its 32 contributions then go out in a few lines.  The
 * units' sizes are scanned (CUB), and one warp per unit copies its ids.
 */
#include <cub/cub.cuh>

#include "ag_units.h"

#define AG_UNITS_BLK 512

__global__ void __launch_bounds__(AG_UNITS_BLK) ag_units_rows_kernel(const uint32_t *off, const uint32_t *outdeg,
                                                                     uint32_t n, AgUnitPlan u)
{
    constexpr uint32_t PER = AG_UNIT_WIN / AG_UNITS_BLK;
    constexpr uint32_t HUB_KEY = AG_UNIT_LONG / 4u + 2u;
    typedef cub::BlockRadixSort<uint16_t, AG_UNITS_BLK, PER, uint32_t> Sort;
    __shared__ typename Sort::TempStorage tmp;
    __shared__ uint32_t list[AG_UNIT_WIN];
    const uint32_t tid = threadIdx.x, lane = tid & 31, r0 = blockIdx.x * AG_UNIT_WIN, nrows = min(AG_UNIT_WIN, n - r0);
    uint16_t key[PER]; /* quads, longest first; places past the last row end up last */
    uint32_t val[PER];
#pragma unroll
    for (uint32_t k = 0; k < PER; ++k) {
        const uint32_t i = tid * PER + k;
        key[k] = 0;
        val[k] = i;
        if (i < nrows) {
            const uint32_t d = off[r0 + i + 1] - off[r0 + i];
            const bool hub = d > u.longest;
            if (hub) {
                atomicAdd(u.cnt, (d - 1u) / AG_BIN_HUB + 1u);
                atomicAdd(u.cnt + 1, 1u);
            }
            key[k] = (uint16_t)(hub ? HUB_KEY : (d + 3u) / 4u + 1u);
            val[k] = i | (hub ? AG_UNIT_HUB : d << 11);
        }
    }
    Sort(tmp).SortDescending(key, val, 0, 10);
#pragma unroll
    for (uint32_t k = 0; k < PER; ++k)
        list[tid * PER + k] = val[k];
    __syncthreads();
    for (uint32_t i = tid; i < ((nrows + 31u) & ~31u); i += AG_UNITS_BLK) {
        uint32_t x = 0;
        if (i < nrows) {
            x = list[i];
            const uint32_t r = r0 + AG_UNIT_ROW(x);
            u.info[r0 + i] = x;
            u.outdeg[r0 + i] = outdeg[r];
            u.posof[r] = r0 + i;
        }
        const uint32_t most = __reduce_max_sync(0xffffffffu, AG_UNIT_LEN(x));
        if (lane == 0) {
            u.ubase[(r0 + i) >> 5] = 32u * ((most + 3u) >> 2);
            if (((most + 3u) >> 2) > u.heavy_quads)
                u.heavy[atomicAdd(u.cnt + 2, 1u)] = (r0 + i) >> 5;
        }
    }
}

__global__ void ag_units_hubs_kernel(const uint32_t *off, uint32_t n, AgUnitPlan u)
{
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t d = off[v + 1] - off[v];
        if (d <= u.longest)
            continue;
        const uint32_t nch = (d - 1u) / AG_BIN_HUB + 1u, first = atomicAdd(u.cnt, nch);
        u.hrow[atomicAdd(u.cnt + 1, 1u)] = first; /* rows in any order */
        for (uint32_t c = 0; c < nch; ++c)
            u.hubs[first + c] = make_uint4((uint32_t)v, c, first,
                                           (min(AG_BIN_HUB, d - c * AG_BIN_HUB) - 1u) | (nch << 11));
    }
}

/* unit k belongs to batch (quads per row and fixed work before it) / batch */
__device__ __forceinline__ uint32_t ag_units_batch(const AgUnitPlan &u, uint32_t k)
{
    return (uint32_t)(((uint64_t)(u.ubase[k] >> 5) + (uint64_t)AG_UNIT_COST * k) / u.batch);
}

__global__ void ag_units_batches_kernel(AgUnitPlan u)
{
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k <= u.nunits; k += gridDim.x * blockDim.x) {
        const uint32_t b1 = k < u.nunits ? ag_units_batch(u, k) : u.nbatch;
        for (uint32_t b = k ? ag_units_batch(u, k - 1) + 1u : 0u; b <= b1; ++b)
            u.bstart[b] = k;
    }
}

/* T, V: uint32_t, uint4 (ids) or float, float4 (weights) */
template <typename T, typename V>
__global__ void __launch_bounds__(256) ag_units_ids_kernel(const uint32_t *off, const T *ids, uint32_t n,
                                                           const AgUnitPlan u, V *out)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    if (blockIdx.x < u.nhub) {
        const uint4 h = u.hubs[blockIdx.x];
        const uint32_t len = (h.w & (AG_BIN_HUB - 1u)) + 1u;
        const T *src = ids + off[h.x] + (size_t)h.y * AG_BIN_HUB;
        T *dst = reinterpret_cast<T *>(out) + (size_t)blockIdx.x * AG_BIN_HUB;
        for (uint32_t i = tid; i < AG_BIN_HUB; i += 256)
            dst[i] = i < len ? src[i] : T(0);
        return;
    }
    const uint32_t k = (blockIdx.x - u.nhub) * 8u + (tid >> 5);
    if (k >= u.nunits)
        return;
    const uint32_t at = 32u * k + lane;
    const uint32_t x = at < n ? u.info[at] : 0u, len = AG_UNIT_LEN(x);
    const T *src = ids + (len ? off[(at & ~(AG_UNIT_WIN - 1u)) + AG_UNIT_ROW(x)] : 0u);
    const uint32_t b0 = u.ubase[k], rounds = (u.ubase[k + 1] - b0) >> 5;
    V *dst = out + (size_t)u.nhub * (AG_BIN_HUB / 4) + b0 + lane;
    for (uint32_t i = 0; i < rounds; ++i, dst += 32) {
        V q;
        q.x = 4u * i < len ? src[4u * i] : T(0);
        q.y = 4u * i + 1u < len ? src[4u * i + 1u] : T(0);
        q.z = 4u * i + 2u < len ? src[4u * i + 2u] : T(0);
        q.w = 4u * i + 3u < len ? src[4u * i + 3u] : T(0);
        *dst = q;
    }
}

extern "C" cudaError_t ag_units_rows(const uint32_t *row_off, const uint32_t *outdeg, uint32_t n, AgUnitPlan *u,
                                     uint32_t *totals_host, cudaStream_t s)
{
    u->nunits = (n + 31u) / 32u;
    size_t tb = 0;
    cudaError_t e = cub::DeviceScan::ExclusiveSum(nullptr, tb, (const uint32_t *)nullptr, (uint32_t *)nullptr,
                                                  (int)u->nunits + 1, s);
    if (e == cudaSuccess)
        e = cudaMallocAsync(&u->tmp, tb ? tb : 16, s);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(u->cnt, 0, 12, s);
    if (e != cudaSuccess)
        return e;
    ag_units_rows_kernel<<<(n + AG_UNIT_WIN - 1u) / AG_UNIT_WIN, AG_UNITS_BLK, 0, s>>>(row_off, outdeg, n, *u);
    e = cub::DeviceScan::ExclusiveSum(u->tmp, tb, u->ubase, u->ubase, (int)u->nunits + 1, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(totals_host, u->cnt, 12, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(totals_host + 3, u->ubase + u->nunits, 4, cudaMemcpyDeviceToHost, s);
    return e == cudaSuccess ? cudaGetLastError() : e;
}

extern "C" uint32_t ag_units_batches(const AgUnitPlan *u, uint64_t quads)
{
    const uint64_t w = quads / 32u + (uint64_t)AG_UNIT_COST * u->nunits;
    return (uint32_t)(w / u->batch) + 1u;
}

extern "C" cudaError_t ag_units_ids(const uint32_t *row_off, const uint32_t *ids, const float *w, uint32_t n,
                                    const AgUnitPlan *u, cudaStream_t s)
{
    if (u->nhub) {
        cudaError_t e = cudaMemsetAsync(u->cnt, 0, 8, s);
        if (e != cudaSuccess)
            return e;
        ag_units_hubs_kernel<<<ag_sm_grid(16), 256, 0, s>>>(row_off, n, *u);
    }
    ag_units_batches_kernel<<<ag_sm_grid(8), 256, 0, s>>>(*u);
    const uint32_t grid = u->nhub + (u->nunits + 7u) / 8u;
    if (grid) {
        ag_units_ids_kernel<<<grid, 256, 0, s>>>(row_off, ids, n, *u, u->ids);
        if (u->w)
            ag_units_ids_kernel<<<grid, 256, 0, s>>>(row_off, w, n, *u, u->w);
    }
    return cudaGetLastError();
}
