/*
 * ag_ppr.cu -- batched personalized PageRank: k <= 64 source vertices solved
 * together as one sparse-matrix x dense-matrix product per pass.
 *
 * Column i is the pull PageRank of the reference (pageRank.c:1026-1069) with
 * the teleport concentrated on source s_i:
 *   c_i[u]  = r_i[u] / out_degree[u]            (0 without out-edges)
 *   s_i[v]  = sum over v's in-edges of c_i[u]    (binary32, stream order)
 *   r_i'[v] = b_i[v] + damp * s_i[v],  b_i[v] = (1 - damp) * N at v = s_i, else 0
 *   err     = |r_i' - r_i| in binary64 against epsilon; stop when no (v, i)
 *             pair changes by >= epsilon
 * and the result is r_i / N, as for the plain kernel.  The teleport mass
 * (1 - damp) * N keeps the un-normalised scale of the reference's ranks, so
 * the same epsilon means the same thing.
 *
 * Layout: contributions and ranks are N x kp binary32, row-major, kp = k
 * rounded up to 8 (whole 32-byte sectors), 64 above 32.  G lanes (8, 16 or 32,
 * for up to 16, 32 or 64 columns) own a destination row, two columns each, so
 * a warp works on 4, 2 or 1 rows.  Each in-edge becomes one coalesced row
 * gather (the per-edge 4-byte random gather of the single-vector kernel
 * becomes a sequential one of up to 256 bytes).  Every column is summed in
 * stream order, so each column is bit-identical to a sequential binary32 loop.
 *
 * The row gathers, 4 kp bytes per in-edge, are the pass's real traffic, from
 * HBM when the contribution matrix is larger than L2.  A row keeps eight in
 * flight, the grid is exactly the resident warps, and the next row's bounds
 * and first ids load while the current row is gathered, so no warp waits on
 * the offsets -> ids -> rows chain between rows.
 *
 * Rows above AG_PPR_HUB in-edges: eight gathers at a time are a chain of
 * memory latencies (about 110 clocks per in-edge), so that one long row
 * outlasts the rest of the pass.  Some warps, as many as those rows' in-edges
 * call for, take them instead, through a ring of 128 row gathers in shared
 * memory (cp.async).  A lane copies and adds only its own two columns, so the
 * ring needs no synchronisation.
 *
 * us per pass at up to 16, 32 and 64 columns, one kernel of 64 columns and
 * eight gathers per row for all -> here: uniform degrees, 500 K vertices and
 * 4 M in-edges 306 -> 74 to 90, 177, the same; 2 M vertices 1180 -> 400 to 440,
 * 684, the same; R-MAT of 300 K vertices and 2.7 M in-edges 1728 -> 380, 432,
 * 512, of 700 K and 8.8 M 4186 -> 1044, 1041, 1220.  In-edges of long rows per
 * warp on the ring, 16384, 4096, 2048, 1024 (R-MAT 300 K, 8 columns): 702,
 * 451, 402, 388; more warps leave the other rows too few.
 *
 * More than 32 columns on a graph whose plan has no hub rows run on a kernel
 * without the ring: its code costs the other rows 5 % there (321 against 306
 * at 500 K vertices).  So do the smallest graphs with rows of some length.
 *
 * The loop stays on the device: after each pass a one-thread kernel counts
 * it and sets a stop flag once no (v, i) pair moved by epsilon; passes that
 * see the flag return at once, and the host reads the flag every
 * AG_PPR_CHECK passes.
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "ag_device.h"
#include "ag_internal.h"

#define AG_PPR_K 64
#define AG_PPR_BLK 256
#define AG_PPR_DEPTH 8 /* row gathers in flight per row: 64 registers, 32
                          resident warps per SM.  AG_PPR_DEPTH=16 in the
                          environment takes sixteen in the kernel without the
                          ring (80 registers, 24 warps): 8.56 against 7.46 ms
                          per pass on ER 2^23, k = 64 */
#define AG_PPR_WARPS 32u      /* resident warps per SM at that depth         */
#define AG_PPR_HUB 512u       /* rows with more in-edges go through the ring */
#define AG_PPR_HUB_SHARE 1024u /* their in-edges per warp that takes them    */
#define AG_PPR_GROUP 8        /* gathers of one cp.async group             */
#define AG_PPR_GROUPS 16      /* groups of the ring                        */
#define AG_PPR_RING (AG_PPR_GROUP * AG_PPR_GROUPS * AG_PPR_K * 4)
#define AG_PPR_CHECK 8  /* passes between host reads of the stop flag */

/* the device-side loop state, written by ag_ppr_close_kernel */
struct AgPprState
{
    uint32_t stop;       /* set once a pass had no active pair */
    uint32_t passes;     /* passes that did work               */
    uint32_t converged;
    uint32_t nhub, hub_next; /* rows in hubs, the next one to take */
    uint32_t pad;
    unsigned long long active_last, hub_edges;
    double err_last;
};

struct AgPprParams
{
    const uint32_t *row_off;
    const uint32_t *ids;
    const uint32_t *outdeg;
    uint32_t N;
    uint32_t k, kp;   /* columns, floats per row              */
    const float *X;   /* contributions of this pass (N x kp) */
    float *Xn;        /* contributions of the next pass      */
    float *R;         /* ranks (N x kp), updated in place    */
    uint32_t *hubs;   /* rows above AG_PPR_HUB in-edges      */
    const uint32_t *src_rows; /* device row of each source (k entries) */
    float base_src;   /* (1 - damp) * N                       */
    float damp;
    double eps;
    unsigned long long *active; /* pairs with |r' - r| >= eps */
    double *err;      /* sum of |r' - r|                      */
    AgPprState *state;
};

/* two columns of row u: x points at the lane's columns of row 0, `stride`
 * bytes between rows (one wide multiply-add per load; as an index into floats
 * the address took more: 82 instead of 73 us a pass at 500 K vertices and 8
 * columns) */
__device__ __forceinline__ float2 ag_ppr_ld_row(const char *x, uint32_t u, uint32_t stride)
{
    float2 v;
    asm("ld.global.nc.L1::no_allocate.v2.f32 {%0,%1}, [%2];"
        : "=f"(v.x), "=f"(v.y)
        : "l"(x + (uint64_t)u * stride));
    return v;
}

/* device rows of the sources */
__global__ void ag_ppr_sources_kernel(const uint32_t *inv, uint32_t *rows, uint32_t k)
{
    const uint32_t i = threadIdx.x;
    if (i < k)
        rows[i] = inv[rows[i]];
}

/* the rows for the ring */
__global__ void __launch_bounds__(256) ag_ppr_hubs_kernel(AgPprParams p)
{
    for (uint32_t v = blockIdx.x * 256u + threadIdx.x; v < p.N; v += gridDim.x * 256u) {
        const uint32_t n = p.row_off[v + 1] - p.row_off[v];
        if (n > AG_PPR_HUB) {
            p.hubs[atomicAdd(&p.state->nhub, 1u)] = v;
            atomicAdd(&p.state->hub_edges, (unsigned long long)n);
        }
    }
}

template <int G> __global__ void __launch_bounds__(AG_PPR_BLK) ag_ppr_init_kernel(AgPprParams p)
{
    const uint32_t g = threadIdx.x % G;
    const uint32_t kp = G == 32 ? AG_PPR_K : p.kp;
    const uint32_t nr = gridDim.x * (AG_PPR_BLK / G);
    if (2 * g >= kp)
        return;
    const uint32_t s0 = 2 * g < p.k ? p.src_rows[2 * g] : 0xFFFFFFFFu;
    const uint32_t s1 = 2 * g + 1 < p.k ? p.src_rows[2 * g + 1] : 0xFFFFFFFFu;
    for (uint32_t v = blockIdx.x * (AG_PPR_BLK / G) + threadIdx.x / G; v < p.N; v += nr) {
        const uint32_t od = p.outdeg[v];
        float2 r, c;
        r.x = (v == s0) ? p.base_src : 0.0f;
        r.y = (v == s1) ? p.base_src : 0.0f;
        c.x = od ? __fdiv_rn(r.x, __uint2float_rn(od)) : 0.0f;
        c.y = od ? __fdiv_rn(r.y, __uint2float_rn(od)) : 0.0f;
        reinterpret_cast<float2 *>(p.R + (size_t)v * kp)[g] = r;
        reinterpret_cast<float2 *>(p.Xn + (size_t)v * kp)[g] = c;
    }
}

/* a lane's two columns */
template <int G> struct AgPprLane
{
    const AgPprParams &p;
    uint32_t g, gl, kp, s0, s1;
    bool in, live0, live1;
    unsigned long long act;
    double err;

    __device__ __forceinline__ AgPprLane(const AgPprParams &q, uint32_t lane) : p(q)
    {
        g = lane % G;
        kp = G == 32 ? AG_PPR_K : p.kp;
        in = G == 32 || 2 * g < kp;
        /* lanes past the row's end load its last columns again: a predicate on
         * every load costs more */
        gl = G == 32 ? g : min(g, kp / 2u - 1u);
        live0 = 2 * g < p.k;
        live1 = 2 * g + 1 < p.k;
        s0 = live0 ? p.src_rows[2 * g] : 0xFFFFFFFFu;
        s1 = live1 ? p.src_rows[2 * g + 1] : 0xFFFFFFFFu;
        act = 0;
        err = 0.0;
    }

    __device__ __forceinline__ float2 rank(uint32_t v) const
    {
        return reinterpret_cast<const float2 *>(p.R + (size_t)v * kp)[gl];
    }

    /* row v's update from its sums */
    __device__ __forceinline__ void finish(uint32_t v, float ax, float ay, uint32_t od, float2 rp)
    {
        float2 rn, cn;
        rn.x = __fadd_rn((v == s0) ? p.base_src : 0.0f, __fmul_rn(p.damp, ax));
        rn.y = __fadd_rn((v == s1) ? p.base_src : 0.0f, __fmul_rn(p.damp, ay));
        if (!live0)
            rn.x = rp.x = 0.0f;
        if (!live1)
            rn.y = rp.y = 0.0f;
        const double e0 = (double)fabsf(__fsub_rn(rn.x, rp.x));
        const double e1 = (double)fabsf(__fsub_rn(rn.y, rp.y));
        err += e0 + e1;
        act += (unsigned long long)((live0 && e0 >= p.eps) ? 1 : 0) + ((live1 && e1 >= p.eps) ? 1 : 0);
        cn.x = od ? __fdiv_rn(rn.x, __uint2float_rn(od)) : 0.0f;
        cn.y = od ? __fdiv_rn(rn.y, __uint2float_rn(od)) : 0.0f;
        if (in) {
            reinterpret_cast<float2 *>(p.R + (size_t)v * kp)[g] = rn;
            reinterpret_cast<float2 *>(p.Xn + (size_t)v * kp)[g] = cn;
        }
    }
};

/* a pass's counts, all threads of a CTA */
__device__ __forceinline__ void ag_ppr_totals(const AgPprParams &p, unsigned long long my_act, double my_err)
{
    __shared__ unsigned long long s_act[AG_PPR_BLK / 32];
    __shared__ double s_err[AG_PPR_BLK / 32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        my_act += __shfl_xor_sync(0xffffffffu, my_act, o);
        my_err += __shfl_xor_sync(0xffffffffu, my_err, o);
    }
    if (lane == 0) {
        s_act[warp] = my_act;
        s_err[warp] = my_err;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long a = 0;
        double er = 0.0;
        for (int w = 0; w < AG_PPR_BLK / 32; ++w) {
            a += s_act[w];
            er += s_err[w];
        }
        if (a)
            atomicAdd(p.active, a);
        if (er != 0.0)
            atomicAdd(p.err, er);
    }
}

/* rows above AG_PPR_HUB in-edges, one at a time on a whole warp (its first G
 * lanes copy and add) */
template <int G> __device__ __forceinline__ void ag_ppr_hub_rows(AgPprLane<G> &c, uint32_t lane, float2 *ring)
{
    const AgPprParams &p = c.p;
    const uint32_t nhub = p.state->nhub;
    for (;;) {
        uint32_t i = 0;
        if (lane == 0)
            i = atomicAdd(&p.state->hub_next, 1u);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= nhub)
            return;
        const uint32_t v = p.hubs[i], b = p.row_off[v], n = p.row_off[v + 1] - b;
        const uint32_t od = p.outdeg[v], ng = (n + AG_PPR_GROUP - 1u) / AG_PPR_GROUP;
        const float2 rp = c.rank(v);
        /* 32 ids of the groups that are issued next, and of the 64 after them */
        uint32_t i0 = 0, i1 = p.ids[b + lane], i2 = p.ids[b + 32u + lane];
        auto issue = [&](uint32_t t) {
            if (t % 4u == 0) {
                const uint32_t j = (t / 4u + 2u) * 32u + lane;
                i0 = i1;
                i1 = i2;
                i2 = j < n ? p.ids[b + j] : 0u;
            }
#pragma unroll
            for (uint32_t q = 0; q < AG_PPR_GROUP; ++q) {
                const uint32_t u = __shfl_sync(0xffffffffu, i0, (t % 4u) * 8u + q);
                if (lane < G && t * AG_PPR_GROUP + q < n)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(
                                     ring + ((t % AG_PPR_GROUPS) * AG_PPR_GROUP + q) * (AG_PPR_K / 2) + c.g)),
                                 "l"(p.X + (size_t)u * c.kp + 2 * c.gl)
                                 : "memory");
            }
        };
        for (uint32_t t = 0; t < AG_PPR_GROUPS - 1; ++t) {
            if (t < ng)
                issue(t);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        float ax = -0.0f, ay = -0.0f;
        for (uint32_t t = 0; t < ng; ++t) {
            if (t + AG_PPR_GROUPS - 1 < ng)
                issue(t + AG_PPR_GROUPS - 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group %0;" ::"n"(AG_PPR_GROUPS - 1) : "memory");
            const float2 *src = ring + (t % AG_PPR_GROUPS) * AG_PPR_GROUP * (AG_PPR_K / 2) + c.g;
            const uint32_t m = n - t * AG_PPR_GROUP;
#pragma unroll
            for (uint32_t q = 0; q < AG_PPR_GROUP; ++q) {
                if (q < m) {
                    const float2 x = src[q * (AG_PPR_K / 2)];
                    ax = __fadd_rn(ax, x.x);
                    ay = __fadd_rn(ay, x.y);
                }
            }
        }
        if (lane < G)
            c.finish(v, ax, ay, od, rp);
    }
}

template <int G> __global__ void __launch_bounds__(AG_PPR_BLK, 4) ag_ppr_pass_kernel(AgPprParams p)
{
    extern __shared__ __align__(16) float2 ring[];
    if (*(volatile const uint32_t *)&p.state->stop)
        return;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    AgPprLane<G> c(p, lane);
    /* the first warp of the first `hw` CTAs takes hub rows, all other warps
     * the rest */
    const uint32_t hw = p.state->nhub
                            ? min(min(p.state->nhub, gridDim.x), (uint32_t)(p.state->hub_edges / AG_PPR_HUB_SHARE) + 1u)
                            : 0u;
    if (warp == 0 && blockIdx.x < hw) {
        ag_ppr_hub_rows<G>(c, lane, ring);
    } else {
        const uint32_t g = c.g;
        const char *x = reinterpret_cast<const char *>(p.X + 2 * c.gl);
        const uint32_t stride = c.kp * 4u;
        const uint32_t gmask = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << (lane - g);
        const uint32_t w = ((blockIdx.x * AG_PPR_BLK + threadIdx.x) >> 5) - min(hw, blockIdx.x + (warp ? 1u : 0u));
        const uint32_t nr = (gridDim.x * (AG_PPR_BLK / 32) - hw) * (32 / G);
        /* row v's bounds and first ids, and row vn's bounds, are loaded one row
         * ahead of their use */
        uint32_t v = w * (32 / G) + lane / G;
        uint32_t b = 0, e = 0, myid = 0;
        if (v < p.N) {
            b = p.row_off[v];
            e = p.row_off[v + 1];
            myid = g < min((uint32_t)G, e - b) ? p.ids[b + g] : 0u;
        }
        uint32_t vn = v + nr, bn = 0, en = 0;
        if (vn < p.N) {
            bn = p.row_off[vn];
            en = p.row_off[vn + 1];
        }
        while (v < p.N) {
            const uint32_t od = p.outdeg[v];
            const float2 rp = c.rank(v);
            const uint32_t myid_n = (vn < p.N && g < min((uint32_t)G, en - bn)) ? p.ids[bn + g] : 0u;
            const uint32_t vnn = vn + nr;
            uint32_t bnn = 0, enn = 0;
            if (vnn < p.N) {
                bnn = p.row_off[vnn];
                enn = p.row_off[vnn + 1];
            }
            if (e - b <= AG_PPR_HUB) {
                /* stream order; -0 + x = x for every binary32 x, so the sum
                 * starts at -0 instead of at the first value, and a row without
                 * in-edges still gives +0 once the teleport term (+0 or
                 * positive) is added */
                float ax = -0.0f, ay = -0.0f;
                for (uint32_t j0 = b; j0 < e; j0 += G) {
                    const uint32_t n = min((uint32_t)G, e - j0);
                    const uint32_t chunk = (j0 == b) ? myid : (g < n ? p.ids[j0 + g] : 0u);
                    for (uint32_t t = 0; t < n; t += AG_PPR_DEPTH) {
                        float2 val[AG_PPR_DEPTH];
#pragma unroll
                        for (int q = 0; q < AG_PPR_DEPTH; ++q) {
                            const uint32_t u = __shfl_sync(gmask, chunk, (t + q) & (G - 1), G);
                            val[q] = (t + q < n) ? ag_ppr_ld_row(x, u, stride) : make_float2(0.f, 0.f);
                        }
#pragma unroll
                        for (int q = 0; q < AG_PPR_DEPTH; ++q) {
                            if (t + q < n) {
                                ax = __fadd_rn(ax, val[q].x);
                                ay = __fadd_rn(ay, val[q].y);
                            }
                        }
                    }
                }
                c.finish(v, ax, ay, od, rp);
            }
            v = vn;
            b = bn;
            e = en;
            myid = myid_n;
            vn = vnn;
            bn = bnn;
            en = enn;
        }
    }
    __syncwarp();
    ag_ppr_totals(p, c.act, c.err);
}

/* 33 to 64 columns on a graph without hub rows: a warp per row, no ring */
__device__ __forceinline__ float2 ag_ppr_ld_row64(const float *X, uint32_t u, uint32_t lane)
{
    float2 v;
    asm("ld.global.nc.L1::no_allocate.v2.f32 {%0,%1}, [%2];"
        : "=f"(v.x), "=f"(v.y)
        : "l"(X + (size_t)u * AG_PPR_K + 2 * lane));
    return v;
}

template <int DEPTH>
__global__ void __launch_bounds__(AG_PPR_BLK) ag_ppr_wide_kernel(AgPprParams p)
{
    __shared__ unsigned long long s_act[AG_PPR_BLK / 32];
    __shared__ double s_err[AG_PPR_BLK / 32];
    if (*(volatile const uint32_t *)&p.state->stop)
        return;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const uint32_t c0 = 2 * lane, c1 = c0 + 1;
    const bool live0 = c0 < p.k, live1 = c1 < p.k;
    const uint32_t s0 = live0 ? p.src_rows[c0] : 0xFFFFFFFFu;
    const uint32_t s1 = live1 ? p.src_rows[c1] : 0xFFFFFFFFu;
    unsigned long long my_act = 0;
    double my_err = 0.0;
    /* row v's bounds and first ids, and row vn's bounds, are loaded one row
     * ahead of their use */
    uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t b = 0, e = 0, myid = 0;
    if (v < p.N) {
        b = p.row_off[v];
        e = p.row_off[v + 1];
        myid = lane < min(32u, e - b) ? p.ids[b + lane] : 0u;
    }
    uint32_t vn = v + nw, bn = 0, en = 0;
    if (vn < p.N) {
        bn = p.row_off[vn];
        en = p.row_off[vn + 1];
    }
    while (v < p.N) {
        const uint32_t od = p.outdeg[v];
        const float2 rp = reinterpret_cast<const float2 *>(p.R + (size_t)v * AG_PPR_K)[lane];
        const uint32_t myid_n = (vn < p.N && lane < min(32u, en - bn)) ? p.ids[bn + lane] : 0u;
        const uint32_t vnn = vn + nw;
        uint32_t bnn = 0, enn = 0;
        if (vnn < p.N) {
            bnn = p.row_off[vnn];
            enn = p.row_off[vnn + 1];
        }
        /* stream order; -0 + x = x for every binary32 x, so the sum starts
         * at -0 instead of at the first value, and a row without in-edges
         * still gives +0 once the teleport term (+0 or positive) is added */
        float ax = -0.0f, ay = -0.0f;
        for (uint32_t j0 = b; j0 < e; j0 += 32) {
            const uint32_t n = min(32u, e - j0);
            const uint32_t chunk = (j0 == b) ? myid : (lane < n ? p.ids[j0 + lane] : 0u);
            for (uint32_t t = 0; t < n; t += DEPTH) {
                float2 val[DEPTH];
#pragma unroll
                for (int q = 0; q < DEPTH; ++q) {
                    const uint32_t u = __shfl_sync(0xffffffffu, chunk, (t + q) & 31);
                    val[q] = (t + q < n) ? ag_ppr_ld_row64(p.X, u, lane) : make_float2(0.f, 0.f);
                }
#pragma unroll
                for (int q = 0; q < DEPTH; ++q) {
                    if (t + q < n) {
                        ax = __fadd_rn(ax, val[q].x);
                        ay = __fadd_rn(ay, val[q].y);
                    }
                }
            }
        }
        float2 rn, cn;
        rn.x = __fadd_rn((v == s0) ? p.base_src : 0.0f, __fmul_rn(p.damp, ax));
        rn.y = __fadd_rn((v == s1) ? p.base_src : 0.0f, __fmul_rn(p.damp, ay));
        if (!live0)
            rn.x = 0.0f;
        if (!live1)
            rn.y = 0.0f;
        const double e0 = (double)fabsf(__fsub_rn(rn.x, rp.x));
        const double e1 = (double)fabsf(__fsub_rn(rn.y, rp.y));
        my_err += e0 + e1;
        my_act += (unsigned long long)((live0 && e0 >= p.eps) ? 1 : 0) + ((live1 && e1 >= p.eps) ? 1 : 0);
        cn.x = od ? __fdiv_rn(rn.x, __uint2float_rn(od)) : 0.0f;
        cn.y = od ? __fdiv_rn(rn.y, __uint2float_rn(od)) : 0.0f;
        reinterpret_cast<float2 *>(p.R + (size_t)v * AG_PPR_K)[lane] = rn;
        reinterpret_cast<float2 *>(p.Xn + (size_t)v * AG_PPR_K)[lane] = cn;
        v = vn;
        b = bn;
        e = en;
        myid = myid_n;
        vn = vnn;
        bn = bnn;
        en = enn;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        my_act += __shfl_xor_sync(0xffffffffu, my_act, o);
        my_err += __shfl_xor_sync(0xffffffffu, my_err, o);
    }
    if (lane == 0) {
        s_act[warp] = my_act;
        s_err[warp] = my_err;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long a = 0;
        double er = 0.0;
        for (int w = 0; w < AG_PPR_BLK / 32; ++w) {
            a += s_act[w];
            er += s_err[w];
        }
        if (a)
            atomicAdd(p.active, a);
        if (er != 0.0)
            atomicAdd(p.err, er);
    }
}

/* after each pass: count it, keep its statistics, stop when nothing moved;
 * clears the counters for the next pass */
__global__ void ag_ppr_close_kernel(AgPprParams p)
{
    AgPprState *st = p.state;
    if (!st->stop) {
        st->passes += 1;
        st->active_last = *p.active;
        st->err_last = *p.err;
        if (*p.active == 0) {
            st->stop = 1;
            st->converged = 1;
        }
    }
    st->hub_next = 0;
    *p.active = 0;
    *p.err = 0.0;
}

/* out[perm[v] * k + i] = R[v][i] / N (binary32), caller order; a warp per row */
__global__ void __launch_bounds__(256) ag_ppr_output_kernel(AgPprParams p, const uint32_t *perm, float *out)
{
    const float fN = __uint2float_rn(p.N);
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t v = (blockIdx.x * 256u + threadIdx.x) >> 5; v < p.N; v += gridDim.x * 8u) {
        const uint32_t dst = perm ? perm[v] : v;
        for (uint32_t i = lane; i < p.k; i += 32)
            out[(size_t)dst * p.k + i] = __fdiv_rn(p.R[(size_t)v * p.kp + i], fN);
    }
}

/* the kernels for k columns */
template <int G> static void ppr_pick(void (**pass)(AgPprParams), void (**init)(AgPprParams), uint32_t *lanes)
{
    *pass = ag_ppr_pass_kernel<G>;
    *init = ag_ppr_init_kernel<G>;
    *lanes = G;
}

/* host side ------------------------------------------------------------ */

extern "C" ag_status_t ag_ppr_spmm(ag_graph_t g, const uint32_t *sources, uint32_t k, uint32_t max_iterations,
                                   double epsilon, float *ranks, ag_pr_result *result)
{
    ag_clear_error();
    AgGraphView gv;
    ag_status_t st = ag_rt_graph_view(g, &gv);
    if (st != AG_OK)
        return st;
    if (!sources || k == 0 || k > AG_PPR_K)
        return ag_set_error(AG_ERR_INVALID_ARG, "ag_ppr_spmm: need 1..%d sources", AG_PPR_K);
    for (uint32_t i = 0; i < k; ++i)
        if (sources[i] >= gv.N)
            return ag_set_error(AG_ERR_INVALID_ARG, "ag_ppr_spmm: source %u >= %u vertices", sources[i], gv.N);
    cudaStream_t s = gv.stream;
    /* Rows that the ring is for, or not.  Without any, a graph of no more rows
     * than resident warps gives each row a warp whatever k, if some rows are
     * long: rows that share a warp wait for the longest of them.  us of five
     * passes, one column, on the shared kernel / so: R-MAT of 1024 vertices
     * (rows of some hundreds) 203 / 177, 600 137 / 127; uniform 1024 (up to 35)
     * 91 / 98, 4500 102 / 105. */
    const bool hub_rows = gv.max_in_degree > AG_PPR_HUB;
    const bool wide = k > 32 || (!hub_rows && gv.max_in_degree > 64 && gv.N <= ag_sm_grid(AG_PPR_WARPS));
    const uint32_t kp = wide ? AG_PPR_K : (k + 7u) & ~7u;
    const size_t mat = (size_t)gv.N * kp * sizeof(float);
    float *X = nullptr, *Xn = nullptr, *R = nullptr, *out = nullptr;
    uint32_t *src_dev = nullptr, *hubs = nullptr;
    unsigned long long *ctr = nullptr;
    AgPprState *state = nullptr;
    AgPprState hs;
    int per_sm = 0;
    void (*pass_kernel)(AgPprParams) = nullptr, (*init_kernel)(AgPprParams) = nullptr;
    uint32_t lanes = 32;
    size_t ring = AG_PPR_RING;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaError_t err = cudaSuccess;
    uint32_t passes = 0, converged = 0;
    unsigned long long act_last = 0;
    double err_last = 0.0;
    float ms = 0.0f;
    AgPprParams p;
    memset(&p, 0, sizeof(p));
    unsigned grid_rows = 1, grid_pass = 1;
    uint64_t row_blocks = 1;
    memset(&hs, 0, sizeof(hs));
#define PCHK(call)                                                                                       \
    do {                                                                                                 \
        err = (call);                                                                                    \
        if (err != cudaSuccess)                                                                          \
            goto done;                                                                                   \
    } while (0)
    PCHK(cudaMallocAsync((void **)&X, mat, s));
    PCHK(cudaMallocAsync((void **)&Xn, mat, s));
    PCHK(cudaMallocAsync((void **)&R, mat, s));
    PCHK(cudaMallocAsync((void **)&src_dev, AG_PPR_K * 4, s));
    PCHK(cudaMallocAsync((void **)&ctr, 16, s));
    PCHK(cudaMallocAsync((void **)&state, sizeof(AgPprState), s));
    PCHK(cudaMemsetAsync(ctr, 0, 16, s));
    PCHK(cudaMemsetAsync(state, 0, sizeof(AgPprState), s));
    if (wide)
        ppr_pick<32>(&pass_kernel, &init_kernel, &lanes);
    else if (k <= 16)
        ppr_pick<8>(&pass_kernel, &init_kernel, &lanes);
    else
        ppr_pick<16>(&pass_kernel, &init_kernel, &lanes);
    if (wide && !gv.long_rows) {
        const char *d = getenv("AG_PPR_DEPTH");
        pass_kernel = (d && atoi(d) == 16) ? ag_ppr_wide_kernel<16> : ag_ppr_wide_kernel<AG_PPR_DEPTH>;
        ring = 0;
    }
    if (!hub_rows)
        ring = 0;
    if (ring)
        PCHK(cudaMallocAsync((void **)&hubs, ((size_t)gv.E / AG_PPR_HUB + 1) * 4, s));
    PCHK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pass_kernel, AG_PPR_BLK, ring));
    /* init: a few waves; passes: exactly the resident CTAs, so that every
     * warp's share of rows runs at once */
    row_blocks = std::max<uint64_t>(1, ((uint64_t)gv.N * lanes + AG_PPR_BLK - 1) / AG_PPR_BLK);
    grid_rows = (unsigned)std::min<uint64_t>(row_blocks, (uint64_t)ag_sm_grid(8));
    grid_pass = (unsigned)std::min<uint64_t>(row_blocks, (uint64_t)ag_sm_grid((unsigned)std::max(per_sm, 1)));
    /* sources in device numbering */
    PCHK(cudaMemcpyAsync(src_dev, sources, (size_t)k * 4, cudaMemcpyHostToDevice, s));
    if (gv.inv)
        ag_ppr_sources_kernel<<<1, AG_PPR_K, 0, s>>>(gv.inv, src_dev, k);
    PCHK(cudaEventCreate(&e0));
    PCHK(cudaEventCreate(&e1));
    p.row_off = gv.row_off;
    p.ids = gv.ids;
    p.outdeg = gv.outdeg;
    p.N = gv.N;
    p.k = k;
    p.kp = kp;
    p.src_rows = src_dev;
    p.hubs = hubs;
    p.damp = Damp;
    p.base_src = (1.0f - Damp) * (float)gv.N; /* one binary32 multiply */
    p.eps = epsilon;
    p.active = ctr;
    p.err = reinterpret_cast<double *>(ctr + 1);
    p.state = state;
    PCHK(cudaEventRecord(e0, s));
    p.X = X;
    p.Xn = X; /* init writes the first contributions into X */
    p.R = R;
    if (ring)
        ag_ppr_hubs_kernel<<<grid_rows, 256, 0, s>>>(p);
    init_kernel<<<grid_rows, AG_PPR_BLK, 0, s>>>(p);
    PCHK(cudaGetLastError());
    for (uint32_t it = 0; it < max_iterations; ++it) {
        p.X = (it & 1) ? Xn : X;
        p.Xn = (it & 1) ? X : Xn;
        pass_kernel<<<grid_pass, AG_PPR_BLK, ring, s>>>(p);
        ag_ppr_close_kernel<<<1, 1, 0, s>>>(p);
        PCHK(cudaGetLastError());
        if ((it + 1) % AG_PPR_CHECK == 0 || it + 1 == max_iterations) {
            PCHK(cudaMemcpyAsync(&hs, state, sizeof(hs), cudaMemcpyDeviceToHost, s));
            PCHK(cudaStreamSynchronize(s));
            if (hs.stop)
                break;
        }
    }
    PCHK(cudaEventRecord(e1, s));
    passes = hs.passes;
    converged = hs.converged;
    act_last = hs.active_last;
    err_last = hs.err_last;
    if (ranks) {
        PCHK(cudaMallocAsync((void **)&out, (size_t)gv.N * k * sizeof(float), s));
        ag_ppr_output_kernel<<<ag_sm_grid(8), 256, 0, s>>>(p, gv.perm, out);
        PCHK(cudaGetLastError());
        st = ag_rt_copy_to_host(ranks, out, (size_t)gv.N * k * sizeof(float));
        if (st != AG_OK)
            goto done;
    }
    PCHK(cudaStreamSynchronize(s));
    cudaEventElapsedTime(&ms, e0, e1);
    if (result) {
        memset(result, 0, sizeof(*result));
        result->passes = passes;
        result->converged = converged;
        result->iterations = converged ? passes - 1 : passes;
        result->active_last = (uint32_t)std::min<unsigned long long>(act_last, 0xFFFFFFFFull);
        result->error_total = err_last / ((double)gv.N * k);
        result->device_ms = ms;
    }
done:
    if (X)
        cudaFreeAsync(X, s);
    if (Xn)
        cudaFreeAsync(Xn, s);
    if (R)
        cudaFreeAsync(R, s);
    if (out)
        cudaFreeAsync(out, s);
    if (src_dev)
        cudaFreeAsync(src_dev, s);
    if (hubs)
        cudaFreeAsync(hubs, s);
    if (ctr)
        cudaFreeAsync(ctr, s);
    if (state)
        cudaFreeAsync(state, s);
    if (e0)
        cudaEventDestroy(e0);
    if (e1)
        cudaEventDestroy(e1);
#undef PCHK
    if (err != cudaSuccess) {
        cudaGetLastError();
        return ag_set_error(AG_ERR_CUDA, "ag_ppr_spmm: %s", cudaGetErrorString(err));
    }
    return st;
}
