/*
 * ag_plan.cu -- device planner of the pull kernel's work lists.
 *
 * Both lists are built from the device row offsets in two walks of the rows:
 * one warp per segment of AG_PLAN_SEG consecutive rows counts its items, the
 * counts are scanned, and a second walk writes every item at its final
 * position.  The lists, the item kinds and their order are those of the
 * pull kernel's contract:
 *   FAST and EXACT (the same list): hub chunks (rows above hub_chunk
 *           in-edges, split in chunks), then long rows (above task_edges),
 *           then row items.  The kernel's order decides how each is summed.
 * A row item packs at most AG_WROWS consecutive rows of at most task_edges
 * in-edges each and together; it never crosses the first row of a graph of
 * a block-diagonal union, nor a segment boundary (a segment holds 512 rows,
 * so the boundary costs at most one extra item per 512 rows).  Within each
 * kind, items follow row order.  Which rows share an item never changes a
 * result: sums depend only on a row's own edges and on the row's kind.
 */
#include <cub/cub.cuh>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "ag_device.h"

#define AG_PLAN_SEG 512u

struct AgPlanArgs
{
    const uint32_t *off;
    const uint32_t *gstart; /* ngraphs + 1 first rows, or NULL */
    uint32_t n, cap, whub, ngraphs, nseg;
};

/* index of the first graph start above row r (ngraphs + 1 when none) */
__device__ __forceinline__ uint32_t ag_plan_next_graph(const AgPlanArgs &a, uint32_t r)
{
    uint32_t lo = 0, hi = a.ngraphs + 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a.gstart[mid] <= r)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

/* A segment is one warp's work.  Its row starts are loaded once (coalesced)
 * into shared memory, and every step places the items of up to 32 rows: the
 * lanes look at the next 32 rows and the first that does not fit ends a row
 * item; a run of longer rows is placed a row per lane.  (One thread per
 * segment walking its rows from memory took 285 us per walk at 1 M rows and
 * 442 at 65 K, where a single CTA was busy; now 89 and 55.)
 * Counts per segment: hub chunks, long rows (not split), row items, split
 * rows.  WRITE = false fills them; WRITE = true reads their exclusive scan
 * and writes the lists. */
#define AG_PLAN_WARPS 4
template <bool WRITE>
__global__ void __launch_bounds__(32 * AG_PLAN_WARPS) ag_plan_kernel(const AgPlanArgs a, uint4 *cnt, const uint4 *scan,
                                                                     AgPlanTotals tot, uint4 *fast, uint4 *exact)
{
    __shared__ uint32_t soff[AG_PLAN_WARPS][AG_PLAN_SEG + 1];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t seg = blockIdx.x * AG_PLAN_WARPS + warp;
    if (seg >= a.nseg)
        return;
    const uint32_t r0 = seg * AG_PLAN_SEG, rows = min(a.n - r0, AG_PLAN_SEG);
    uint32_t *off = soff[warp];
    for (uint32_t i = lane; i <= rows; i += 32)
        off[i] = a.off[r0 + i];
    __syncwarp();
    uint32_t nh = 0, nl = 0, nw = 0, nhr = 0;
    uint4 base = make_uint4(0, 0, 0, 0);
    if (WRITE)
        base = scan[seg];
    uint32_t gi = a.gstart ? ag_plan_next_graph(a, r0) : 0;
    uint32_t r = 0; /* row of the segment */
    while (r < rows) {
        const uint32_t o0 = off[r];
        if (off[r + 1] - o0 > a.cap) {
            /* the rows above cap from here on, one per lane */
            const uint32_t x = r + lane;
            uint32_t d = 0, ox = 0;
            if (x < rows) {
                ox = off[x];
                d = off[x + 1] - ox;
            }
            const uint32_t no = ~__ballot_sync(0xffffffffu, d > a.cap);
            const uint32_t run = no ? (uint32_t)__ffs(no) - 1u : 32u;
            const bool mine = lane < run, hub = mine && d > a.whub;
            const uint32_t nch = hub ? (d - 1u) / a.whub + 1u : 0u;
            const uint32_t hubs = __ballot_sync(0xffffffffu, hub), longs = __ballot_sync(0xffffffffu, mine && !hub);
            uint32_t inc = nch;
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o)
                    inc += t;
            }
            if (WRITE) {
                const uint32_t pbase = base.x + nh + inc - nch;
                for (uint32_t c = 0; c < nch; ++c) {
                    const uint32_t cb = ox + c * a.whub;
                    const uint4 it = make_uint4((AG_T_HUB << 30) | (r0 + x), pbase | (c << AG_SLOT_BITS), cb,
                                                cb + min(ox + d - cb, a.whub));
                    fast[pbase + c] = it;
                    exact[pbase + c] = it;
                }
                if (mine && !hub) {
                    const uint32_t k = tot.hub_items + base.y + nl + __popc(longs & ((1u << lane) - 1u));
                    const uint4 lng = make_uint4((AG_T_LONG << 30) | (r0 + x), r0 + x + 1, ox, ox + d);
                    fast[k] = lng;
                    exact[k] = lng;
                }
            }
            nh += __shfl_sync(0xffffffffu, inc, 31);
            nl += __popc(longs);
            nhr += __popc(hubs);
            r += run;
            continue;
        }
        /* a row item: the first row always fits (d <= cap) */
        uint32_t limit = rows;
        if (a.gstart) {
            while (gi <= a.ngraphs && a.gstart[gi] <= r0 + r)
                ++gi;
            if (gi <= a.ngraphs)
                limit = min(limit, a.gstart[gi] - r0);
        }
        const uint32_t x = r + lane;
        const bool fits = x < limit && off[x + 1] - off[x] <= a.cap && off[x + 1] - o0 <= a.cap;
        const uint32_t no = ~__ballot_sync(0xffffffffu, fits);
        const uint32_t end = r + (no ? (uint32_t)__ffs(no) - 1u : 32u);
        if (WRITE && lane == 0) {
            const uint4 it = make_uint4((AG_T_ROWS << 30) | (r0 + r), r0 + end, o0, off[end]);
            fast[tot.hub_items + tot.long_items + base.z + nw] = it;
            exact[tot.hub_items + tot.long_items + base.z + nw] = it;
        }
        ++nw;
        r = end;
    }
    if (!WRITE && lane == 0)
        cnt[seg] = make_uint4(nh, nl, nw, nhr);
}

struct AgPlanAdd
{
    __device__ __forceinline__ uint4 operator()(const uint4 &a, const uint4 &b) const
    {
        return make_uint4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
    }
};

static AgPlanArgs plan_args(const AgPlanState *ps)
{
    AgPlanArgs a;
    a.off = ps->row_off;
    a.gstart = ps->gstart;
    a.n = ps->n;
    a.cap = ps->cap;
    a.whub = ps->whub;
    a.ngraphs = ps->ngraphs;
    a.nseg = ps->nseg;
    return a;
}

extern "C" void ag_plan_release(AgPlanState *ps, cudaStream_t s)
{
    if (ps->scratch)
        cudaFreeAsync(ps->scratch, s);
    ps->scratch = nullptr;
}

extern "C" cudaError_t ag_plan_count(const uint32_t *row_off, uint32_t n, uint32_t cap, uint32_t whub,
                                     const uint32_t *gstart, uint32_t ngraphs, AgPlanState *ps,
                                     uint32_t *totals_host, cudaStream_t s)
{
    memset(ps, 0, sizeof(*ps));
    ps->row_off = row_off;
    ps->n = n;
    ps->cap = cap;
    ps->whub = whub;
    ps->gstart = gstart;
    ps->ngraphs = gstart ? ngraphs : 0;
    ps->nseg = (n + AG_PLAN_SEG - 1) / AG_PLAN_SEG;
    if (n == 0) {
        memset(totals_host, 0, 4 * sizeof(uint32_t));
        return cudaSuccess;
    }
    const size_t n4 = (size_t)ps->nseg + 1;
    size_t tmp_bytes = 0;
    cudaError_t err = cub::DeviceScan::ExclusiveScan(nullptr, tmp_bytes, (const uint4 *)nullptr, (uint4 *)nullptr,
                                                     AgPlanAdd(), make_uint4(0, 0, 0, 0), (int)n4, s);
    if (err != cudaSuccess)
        return err;
    tmp_bytes = (tmp_bytes + 255) & ~(size_t)255;
    if ((err = cudaMallocAsync(&ps->scratch, 2 * n4 * sizeof(uint4) + tmp_bytes, s)) != cudaSuccess)
        return err;
    void *tmp = ps->scratch; /* scan scratch first: 256-byte aligned */
    uint4 *cnt = reinterpret_cast<uint4 *>(reinterpret_cast<unsigned char *>(ps->scratch) + tmp_bytes);
    ps->scan = cnt + n4;
    if ((err = cudaMemsetAsync(cnt + ps->nseg, 0, sizeof(uint4), s)) != cudaSuccess)
        return err;
    AgPlanTotals none = {0, 0, 0, 0};
    ag_plan_kernel<false><<<(ps->nseg + AG_PLAN_WARPS - 1) / AG_PLAN_WARPS, 32 * AG_PLAN_WARPS, 0, s>>>(
        plan_args(ps), cnt, nullptr, none, nullptr, nullptr);
    err = cub::DeviceScan::ExclusiveScan(tmp, tmp_bytes, cnt, ps->scan, AgPlanAdd(), make_uint4(0, 0, 0, 0), (int)n4, s);
    if (err != cudaSuccess || (err = cudaGetLastError()) != cudaSuccess)
        return err;
    return cudaMemcpyAsync(totals_host, ps->scan + ps->nseg, 4 * sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
}

extern "C" cudaError_t ag_plan_write(AgPlanState *ps, const uint32_t *totals, uint4 *fast, uint4 *exact,
                                     cudaStream_t s)
{
    if (ps->n == 0)
        return cudaSuccess;
    AgPlanTotals tot = {totals[0], totals[1], totals[2], totals[3]};
    ag_plan_kernel<true><<<(ps->nseg + AG_PLAN_WARPS - 1) / AG_PLAN_WARPS, 32 * AG_PLAN_WARPS, 0, s>>>(
        plan_args(ps), nullptr, ps->scan, tot, fast, exact);
    return cudaGetLastError();
}

__global__ void ag_set_u32_kernel(uint32_t *p, uint32_t v) { *p = v; }

/* one 32-bit store on the stream (used for the closing row offset) */
extern "C" cudaError_t ag_set_u32(uint32_t *p, uint32_t v, cudaStream_t s)
{
    ag_set_u32_kernel<<<1, 1, 0, s>>>(p, v);
    return cudaGetLastError();
}
