/*
 * ag_solve.cu -- a whole PageRank pull solve in one cooperative launch.
 *
 * One pull pass (the reference's host contribution loop pageRank.c:1026-1033,
 * its gather on the accelerator and its host update loop pageRank.c:1055-1069):
 *
 *   s[v]  = c[u0] + c[u1] + ...     over v's inverse row, binary32
 *   r'[v] = base + damp * s[v]      binary32 multiply, then add (no FMA)
 *   err   = |r'[v] - r[v]|          binary32 subtract, compared in binary64
 *   c'[v] = r'[v] / out_degree[v]   next pass's contribution (0 if no out-edge)
 *
 * The kernel holds one CTA on every SM and runs the first contributions, every
 * pass and the normalisation, with a grid barrier between them: the last CTA
 * to arrive closes the pass (record, stop test) and releases the others.
 *
 * Bins (ag_bins.h; graphs up to AG_UNIT_MIN_EDGES, and unions).  A CTA's warps
 * form AG_SUBS groups, each with its own shared-memory buffer.  A group takes
 * one bin at a time (hub chunks first, then row bins in row order, handed out
 * by an atomic counter):
 *   stage   every thread loads four slot ids at a time and gathers their
 *           contributions into the buffer, from the CTA's copy of the most-read
 *           ones (hot table) or from L1 / L2;
 *   sum     one row per lane from the buffer, so that 32 rows' stream-order
 *           chains of binary32 adds run side by side;
 *   update  the group's rows in row order, coalesced.
 * While one group waits for its gathers the other sums.
 *
 * Units (ag_units.h; larger graphs).  A warp takes 32 rows of about the same
 * length, one per lane; each lane gathers eight values of its row at a time
 * into registers and adds them in stream order, while the next ids travel.
 * No warp waits for another inside a pass.  Items are handed out by one atomic
 * counter, those with the longest chains first.
 *
 * EXACT order: every row is summed in stream order (a hub row as described at
 * ag_sv_moves).  FAST order: rows of up to 32 in-edges in stream order; longer
 * ones as binary32 trees of eight values added in binary64.
 * Data-driven passes (the reference's worklist pull, pageRank.c:2810-2969): a
 * vertex that changes writes its next contribution with the sign bit set; a
 * row sums magnitudes and is on the worklist when the pass is the first or a
 * sign was set.
 * No result depends on which warp ran what.
 * SpMV: one such pass over any vector.  The launch first puts x into device
 * order (a grid barrier follows), reads the weights in the order of the ids,
 * and writes y in caller order.
 *
 * What bounds a pass: on a small graph the chain of waits (barrier, bin, ids,
 * gathers, the longest row's adds, update), about 7 us at 1024 vertices, where
 * the pull kernel's loop, one launch per pass, took 14.5 (EXACT); from a
 * million in-edges on the gathers' L1 misses (about one per SM clock), and in
 * EXACT order what the hub rows add.  us per pass, FAST and EXACT, pull
 * kernel's loop -> here (R-MAT, 16 edges per vertex): 65 K vertices 19.9 ->
 * 12.9 and 53.8 -> 17.3; 1 M 65.9 -> 66.3 and 127 -> 71.6; 2 M 115 -> 98 and
 * 190 -> 125; 4 M 221 -> 183 and 328 -> 232; 8 M 473 -> 380 and 718 -> 470;
 * 16 M 922 -> 778 and 1332 -> 897 (4E + 24N bytes: 17 -> 25 % of the measured
 * copy rate).  The pull kernel's EXACT order
 * adds a long row on one lane while the other 31 wait; here they add other
 * rows, and neighbouring rows' warps share L1 lines.
 *
 * SpMV, weighted, us per product, FAST and EXACT, as three launches (permute,
 * product by rows of a task, permute) -> here: R-MAT 65 K vertices 33 -> 15.4
 * and 66 -> 29; 1 M 93 -> 70 and 147 -> 97; 4 M 316 -> 222 and 443 -> 336;
 * uniform degrees, 1.2 M 74 -> 70 and 82 -> 72; 4 M 207 -> 190 and 224 -> 190.
 * The weights are 4 more streamed bytes per edge (8E + 20N bytes at the copy
 * rate: 95 us at R-MAT 4 M); the gathers still bound it.
 */
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ag_mem.h"
#include "ag_solve.h"

/* ------------------------------------------------ TMA bulk copy to smem */
__device__ __forceinline__ uint32_t ag_sv_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ag_sv_mbar_init(uint64_t *bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ag_sv_smem(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

/* bounded wait for the mbarrier phase to complete; false if the limit ran out first */
__device__ __forceinline__ bool ag_sv_mbar_wait(uint64_t *bar, uint32_t phase, uint32_t limit)
{
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(ag_sv_smem(bar)), "r"(phase)
                     : "memory");
        if (done)
            return true;
    }
    return false;
}

/* ----------------------------------------------------- element types */
template <int PREC> __device__ __forceinline__ float ag_sv_low(uint16_t h)
{
    return PREC == 1 ? __uint_as_float(((uint32_t)h) << 16) : __half2float(__ushort_as_half(h));
}

template <int PREC> __device__ __forceinline__ uint16_t ag_sv_to_low(float f)
{
    return PREC == 1 ? __bfloat16_as_ushort(__float2bfloat16_rn(f)) : __half_as_ushort(__float2half_rn(f));
}

/* contributions change between the passes of one launch, so their loads are
 * coherent ones (the grid barrier's acquire drops stale L1 lines); ids of the
 * warm tier may take L1 lines, colder ones do not */
__device__ __forceinline__ float ag_sv_ld_f32(const float *p, uint64_t pol, bool l1)
{
    float v;
    if (l1)
        asm volatile("ld.global.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
    else
        asm volatile("ld.global.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
    return v;
}

__device__ __forceinline__ uint16_t ag_sv_ld_u16(const uint16_t *p, uint64_t pol, bool l1)
{
    uint16_t v;
    if (l1)
        asm volatile("ld.global.L2::cache_hint.u16 %0, [%1], %2;" : "=h"(v) : "l"(p), "l"(pol));
    else
        asm volatile("ld.global.L1::no_allocate.L2::cache_hint.u16 %0, [%1], %2;" : "=h"(v) : "l"(p), "l"(pol));
    return v;
}

__device__ __forceinline__ double ag_sv_warp_d(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void ag_sv_sub_sync(uint32_t sub)
{
    asm volatile("bar.sync %0, %1;" ::"r"(sub + 1u), "r"((uint32_t)AG_SUB_THREADS) : "memory");
}

/* a row of `sums` that belongs to a hub row, written by its composer */
#define AG_SV_HUB 0xFFBADBADu

extern __shared__ __align__(128) unsigned char ag_sv_dyn[];

struct AgSvShared
{
    double redd[AG_SOLVE_BLK / 32];
    uint32_t redu[AG_SOLVE_BLK / 32];
    uint64_t mbar;
    uint32_t last, gen, next[AG_SUBS];
    uint16_t pred[AG_SUBS][16 * AG_BIN_ROUNDS + 1];
};

/* ------------------------------------------------------------ exact sums */
/* 2^(150-e) for a biased exponent e in [24, 254] */
__device__ __forceinline__ float ag_sv_scale(uint32_t e) { return __uint_as_float((277u - e) << 23); }

/* s rebuilt from its exponent bits and M (M in [2^23, 2^24)) */
__device__ __forceinline__ float ag_sv_make(uint32_t ex, uint32_t m)
{
    return __uint_as_float((ex << 23) | (m & 0x7fffffu));
}

/* EXACT order of a hub row: the stream-order binary32 sum of up to millions
 * of values, bit for bit, without one chain of that many adds.
 *
 * While s is a positive normal number M * 2^(e-150), adding v >= 0 moves M by
 * an integer: with x = v / 2^(e-150) and f = floor(x), the binary32 add gives
 * M + f, M + f + 1 above the half, and the even one of the two at a tie, which
 * M's parity decides.  So a run of adds is a map of M known from two numbers,
 * how far it moves an even M and how far an odd one, as long as M stays below
 * 2^24 (the moves are never negative).  Such maps compose, and composition is
 * associative: a lane composes eight consecutive values, a shuffle scan the
 * lanes of a round, and the composing warp the rounds.
 *
 * moves of this lane's eight values v at exponent e: d[0] of an even, d[1] of
 * an odd M; a value that is negative, not finite or 2^22 units or more makes
 * both 2^24 (M leaves the binade) */
__device__ __forceinline__ void ag_sv_moves(const float *v, uint32_t e, uint32_t &d0, uint32_t &d1)
{
    const float sc = ag_sv_scale(e);
    bool leaves = false;
    d0 = d1 = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float x = __fmul_rn(v[i], sc);
        leaves |= !((x >= 0.0f) & (x < 4194304.0f));
        /* floor(x) in the low bits of 2^23 + x, and the rest */
        const float y = __fadd_rd(x, 8388608.0f);
        const float fr = __fsub_rn(x, __fsub_rn(y, 8388608.0f));
        const uint32_t k = (__float_as_uint(y) & 0x7fffffu) + (fr > 0.5f ? 1u : 0u);
        const uint32_t tie = fr == 0.5f ? 1u : 0u;
        d0 += k;
        d0 += d0 & tie;
        d1 += k;
        d1 += ~d1 & tie;
    }
    if (leaves)
        d0 = d1 = 1u << 24;
}

/* inclusive scan of the lanes' maps (totals of 2^24 or more stay 2^24) */
__device__ __forceinline__ void ag_sv_scan(uint32_t lane, uint32_t &d0, uint32_t &d1)
{
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t u0 = __shfl_up_sync(0xffffffffu, d0, o), u1 = __shfl_up_sync(0xffffffffu, d1, o);
        if (lane >= o) {
            const uint32_t n0 = u0 + ((u0 & 1u) ? d1 : d0), n1 = u1 + ((u1 & 1u) ? d0 : d1);
            d0 = min(n0, 1u << 24);
            d1 = min(n1, 1u << 24);
        }
    }
}

/* a lane's eight consecutive values of a round in shared memory */
template <int MODE>
__device__ __forceinline__ void ag_sv_eight(const float *vals, uint32_t n, uint32_t lane, float *v)
{
    const uint32_t j = 8u * lane;
    const float4 q0 = *reinterpret_cast<const float4 *>(vals + j), q1 = *reinterpret_cast<const float4 *>(vals + j + 4);
    v[0] = q0.x, v[1] = q0.y, v[2] = q0.z, v[3] = q0.w;
    v[4] = q1.x, v[5] = q1.y, v[6] = q1.z, v[7] = q1.w;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (MODE == AG_MODE_DD)
            v[i] = fabsf(v[i]);
        if (j + i >= n)
            v[i] = 0.0f; /* s + 0 = s: s is positive here */
    }
}

/* the stream-order sum of vals[0, n) by one lane, continuing s (s = -0 starts
 * a sum: -0 + x = x); the next eight values load while eight are added */
template <int MODE> __device__ __forceinline__ float ag_sv_chain(const float *vals, uint32_t n, float s)
{
    const float4 *q = reinterpret_cast<const float4 *>(vals);
    auto mag = [](float x) { return MODE == AG_MODE_DD ? fabsf(x) : x; };
    float4 a = q[0], b = q[1];
    uint32_t j = 0;
    for (; j + 8u <= n; j += 8u) {
        q += 2;
        const float4 na = q[0], nb = q[1];
        s = __fadd_rn(s, mag(a.x));
        s = __fadd_rn(s, mag(a.y));
        s = __fadd_rn(s, mag(a.z));
        s = __fadd_rn(s, mag(a.w));
        s = __fadd_rn(s, mag(b.x));
        s = __fadd_rn(s, mag(b.y));
        s = __fadd_rn(s, mag(b.z));
        s = __fadd_rn(s, mag(b.w));
        a = na;
        b = nb;
    }
    const float t[7] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z};
#pragma unroll
    for (int i = 0; i < 7; ++i)
        if (j + i < n)
            s = __fadd_rn(s, mag(t[i]));
    return s;
}

/* FAST order of a row above AG_BIN_SEQ in-edges: trees of eight values, added
 * in binary64.  Data-driven: `tag` gets the values' sign bits (its other bits
 * mean nothing; read in a loop of their own they took 15 us of a pass at 1 M
 * R-MAT vertices: 78.5 -> 63.3) */
template <int MODE> __device__ __forceinline__ float ag_sv_fast(const float *vals, uint32_t n, uint32_t &tag)
{
    const float4 *q = reinterpret_cast<const float4 *>(vals);
    auto mag = [&](float x) {
        if (MODE != AG_MODE_DD)
            return x;
        tag |= __float_as_uint(x);
        return fabsf(x);
    };
    /* two sums, so that one eight's tree runs while the other is added */
    double t = 0.0, t1 = 0.0;
    auto eight = [&](float4 a, float4 b) {
        const float x = __fadd_rn(__fadd_rn(mag(a.x), mag(a.y)), __fadd_rn(mag(a.z), mag(a.w)));
        const float y = __fadd_rn(__fadd_rn(mag(b.x), mag(b.y)), __fadd_rn(mag(b.z), mag(b.w)));
        return (double)__fadd_rn(x, y);
    };
    uint32_t j = 0;
    for (; j + 16u <= n; j += 16u, q += 4) {
        const float4 a = q[0], b = q[1], c = q[2], d = q[3];
        t += eight(a, b);
        t1 += eight(c, d);
    }
    for (; j < n; j += 8u, q += 2) {
        float4 a = q[0], b = q[1];
        if (j + 8u > n) {
            const uint32_t m = n - j; /* 1 .. 7 */
            if (m < 2) a.y = 0.0f;
            if (m < 3) a.z = 0.0f;
            if (m < 4) a.w = 0.0f;
            if (m < 5) b.x = 0.0f;
            if (m < 6) b.y = 0.0f;
            if (m < 7) b.z = 0.0f;
            b.w = 0.0f;
        }
        t += eight(a, b);
    }
    t += t1;
    return __double2float_rn(t);
}

/* one round of a hub row on the whole warp: the stream-order sum of 256
 * values, eight consecutive ones per lane (0 past the row's end), continuing s
 * (the same in every lane, as is the result).  The lane where s leaves its
 * binade adds its own eight values in binary32, and the lanes after it start
 * again in the new binade. */
__device__ __noinline__ float ag_sv_round(float v0, float v1, float v2, float v3, float v4, float v5, float v6, float v7,
                                          float s, uint32_t lane, uint32_t done)
{
    const float v[8] = {v0, v1, v2, v3, v4, v5, v6, v7};
    while (done < 32u) { /* lanes below `done` are in s */
        const uint32_t sb = __float_as_uint(s), ex = sb >> 23;
        uint32_t out = done;
        if (ex >= 24u && ex <= 254u) {
            const uint32_t m = (sb & 0x7fffffu) | 0x800000u;
            uint32_t d0 = 0, d1 = 0;
            if (lane >= done)
                ag_sv_moves(v, ex, d0, d1);
            ag_sv_scan(lane, d0, d1);
            const uint32_t to = m + ((m & 1u) ? d1 : d0);
            const uint32_t ok = __ballot_sync(0xffffffffu, to < (1u << 24));
            if (ok == 0xffffffffu)
                return ag_sv_make(ex, __shfl_sync(0xffffffffu, to, 31));
            out = __ffs(~ok) - 1;
            const uint32_t before = __shfl_sync(0xffffffffu, to, (out - 1u) & 31u);
            s = ag_sv_make(ex, out ? before : m);
        } /* else zero, tiny, negative or not finite: one lane after another */
#pragma unroll
        for (int i = 0; i < 8; ++i)
            s = __fadd_rn(s, v[i]);
        s = __shfl_sync(0xffffffffu, s, out);
        done = out + 1;
    }
    return s;
}

/* a round's map in one word: the move of an even M, and the odd one's
 * difference (it is -1, 0 or 1) + 1 in bits 26 and 27; AG_XNOT: does not apply */
__device__ __forceinline__ uint32_t ag_sv_pack(uint32_t d0, uint32_t d1)
{
    return d0 >= (1u << 24) || d1 >= (1u << 24) ? AG_XNOT : d0 | ((d1 + 1u - d0) << 26);
}

/* Each round is mapped at two neighbouring exponents, this one and the next:
 * those nearest to where its sum began in the pass before (`pred`, the top
 * half of its bits), so that a sum that moved by less than 41 % still finds
 * its map, or the two that it passes through when the round after it began
 * (`next`) in a higher binade */
__device__ __forceinline__ uint32_t ag_sv_low_exp(uint32_t pred, uint32_t next)
{
    const uint32_t e = pred >> 7;
    return (pred & 0x7fu) >= 53u || (next >> 7) > e || e == 0u ? e : e - 1u;
}

#define AG_SV_NOT_KEPT 0xffffffffu

/* values of a hub row added one by one (N consecutive ones per lane, lanes
 * below `done` are in s), one lane after another */
template <int N> __device__ __forceinline__ float ag_sv_serial(const float *v, float s, uint32_t done)
{
#pragma unroll 4
    for (; done < 32u; ++done) {
#pragma unroll
        for (int i = 0; i < N; ++i)
            s = __fadd_rn(s, v[i]);
        s = __shfl_sync(0xffffffffu, s, done);
    }
    return s;
}

/* the arrival word, no CTA there yet, of the barrier after barrier word gen */
__device__ __forceinline__ uint32_t ag_sv_arrivals(uint32_t gen)
{
    return (gen >> AG_GEN_SHIFT) * (AG_COUNT_CTAS + 1u) & ~AG_COUNT_ABORT;
}

/* One thread of a CTA that waited in vain for barrier word `gen` to change, or
 * found that another did, and runs nothing more.  The arrival word decides how
 * the barrier ends: unless all have arrived it is marked as given up, and
 * nobody opens it any more.  If all have, it opens, and the next one, which
 * this CTA will not reach, is given up instead.  (Called at the kernel's end:
 * a call inside the barrier, even of a function of its own, made passes of
 * FAST bins 1.5 % longer.) */
__device__ __noinline__ void ag_sv_give_up(uint32_t *sync, uint32_t gen, uint32_t ctas, volatile uint32_t *gave_up)
{
    const uint32_t c = ag_sv_arrivals(gen);
    uint32_t now = *((volatile uint32_t *)(sync + AG_SYNC_COUNT));
    bool mine = false;
    /* (at most one round for each CTA that arrives meanwhile) */
    while (!mine && now - c < ctas) {
        const uint32_t was = atomicCAS(sync + AG_SYNC_COUNT, now, now | AG_COUNT_ABORT);
        mine = was == now;
        now = was;
    }
    if (!mine && now < AG_COUNT_ABORT) {
        uint32_t g = gen;
        for (uint32_t i = 0; g == gen && i < 1u << 20; ++i)
            asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(g) : "l"(sync + AG_SYNC_GEN) : "memory");
        atomicOr(sync + AG_SYNC_COUNT, AG_COUNT_ABORT);
    }
    atomicOr(sync + AG_SYNC_GEN, AG_GEN_ABORT);
    *gave_up = 1u;
    __threadfence_system();
}

/* ------------------------------------------------------------------ solve */
template <int MODE, int PREC, bool EXACT, bool UNITS> struct AgSolve
{
    const AgSolveParams &q;
    const AgPullParams &p;
    AgSvShared &sh;
    uint64_t pol_first, pol_last;
    const float *c_in32;
    const uint16_t *c_in16;
    float *c_out32;
    uint16_t *c_out16;
    const float *hot32;
    const uint16_t *hot16;
    uint32_t hot_n;
    uint32_t iter, flags;  /* this pass; AG_GEN_* of the barrier before it */
    uint32_t gen;          /* last value of the barrier word seen          */
    uint32_t mphase;       /* mbarrier phase of the next hot-table copy    */
    double eps, my_err;
    uint32_t my_active;
    uint32_t tid, lane, sub, st, sw; /* thread, lane; group, thread and warp of it */

    __device__ __forceinline__ AgSolve(const AgSolveParams &qq, AgSvShared &s) : q(qq), p(qq.p), sh(s)
    {
        tid = threadIdx.x;
        lane = tid & 31;
        sub = tid / AG_SUB_THREADS;
        st = tid % AG_SUB_THREADS;
        sw = st >> 5;
        pol_first = ag_policy_evict_first();
        pol_last = ag_policy_evict_last();
        my_err = 0.0;
        my_active = 0;
        mphase = 0;
    }

    __device__ __forceinline__ bool low() const { return PREC != 0 && (flags & AG_GEN_READ_LOW); }

    /* ------------------------------------------------------ grid barrier */
    /* every CTA's earlier writes are visible to every CTA after it; `close`
     * runs on the last CTA to arrive (all its threads) and returns the flags
     * that the barrier hands on.  The wait is bounded: a CTA that waits in
     * vain gets false, runs nothing more and gives the barrier up for all
     * (ag_sv_give_up): every other CTA, late ones too, then gets false here or
     * at the kernel's start. */
    template <typename F> __device__ __forceinline__ bool grid_sync(F close)
    {
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            const uint32_t c = atomicAdd(q.sync + AG_SYNC_COUNT, 1u);
            sh.last = (c & (AG_COUNT_ABORT | AG_COUNT_CTAS)) == gridDim.x - 1 ? 1u : 0u;
        }
        __syncthreads();
        if (sh.last) {
            __threadfence();
            const uint32_t f = close();
            if (tid == 0) {
                const uint32_t g = (((gen >> AG_GEN_SHIFT) + 1u) << AG_GEN_SHIFT) | f;
                q.sync[AG_SYNC_COUNT] = ag_sv_arrivals(g);
                q.sync[AG_SYNC_BIN] = 0;
                q.sync[AG_SYNC_KEPT] = 0;
                sh.gen = g;
                asm volatile("fence.acq_rel.gpu;" ::: "memory");
                asm volatile("st.release.gpu.u32 [%0], %1;" ::"l"(q.sync + AG_SYNC_GEN), "r"(g) : "memory");
            }
        } else if (tid == 0) {
            uint32_t g = gen;
            for (uint32_t i = 0; g == gen && i < q.spins; ++i)
                asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(g) : "l"(q.sync + AG_SYNC_GEN) : "memory");
            sh.gen = MODE != AG_MODE_MULTI && g == gen ? gen | AG_GEN_ABORT : g;
            __threadfence();
        }
        __syncthreads();
        /* a wait in vain: the mark in `gen`, in a union the word as it was (either
         * form in all kernels made unions' or FAST passes 2 to 3 % longer) */
        const bool stuck = MODE == AG_MODE_MULTI && sh.gen == gen;
        gen = sh.gen;
        flags = gen & 7u;
        return !stuck && !(gen & AG_GEN_ABORT);
    }

    /* the end of a launch without a closing barrier: the last CTA to get here
     * clears the counters */
    __device__ __forceinline__ void leave()
    {
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            const uint32_t c = atomicAdd(q.sync + AG_SYNC_COUNT, 1u);
            if ((c & AG_COUNT_CTAS) == gridDim.x - 1) {
                q.sync[AG_SYNC_COUNT] = c & ~AG_COUNT_CTAS;
                q.sync[AG_SYNC_BIN] = 0;
                q.sync[AG_SYNC_KEPT] = 0;
                __threadfence();
            }
        }
    }

    /* ------------------------------------------------------------ gathers */
    __device__ __forceinline__ void start_pass()
    {
        const bool odd = (iter & 1u) != 0;
        c_in32 = MODE == AG_MODE_SPMV ? p.x : odd ? p.c32_1 : p.c32_0;
        c_out32 = odd ? p.c32_0 : p.c32_1;
        c_in16 = odd ? p.c16_1 : p.c16_0;
        c_out16 = odd ? p.c16_0 : p.c16_1;
        hot_n = p.hot_n ? (low() ? p.hot_n16 : p.hot_n) : 0u;
        if (tid == 0 && hot_n) {
            /* hot table: the first hot_n contributions, one TMA bulk copy per
             * 32 KB.  They were written through the generic proxy. */
            const uint32_t bytes = hot_n * (low() ? 2u : 4u);
            const unsigned char *src = low() ? (const unsigned char *)c_in16 : (const unsigned char *)c_in32;
            asm volatile("fence.proxy.async;" ::: "memory");
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(ag_sv_smem(&sh.mbar)), "r"(bytes)
                         : "memory");
            for (uint32_t off = 0; off < bytes; off += AG_BULK_CHUNK)
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                 ag_sv_smem(ag_sv_dyn + off)),
                             "l"(src + off), "r"(min(AG_BULK_CHUNK, bytes - off)), "r"(ag_sv_smem(&sh.mbar))
                             : "memory");
        }
        hot32 = reinterpret_cast<const float *>(ag_sv_dyn);
        hot16 = reinterpret_cast<const uint16_t *>(ag_sv_dyn);
    }

    __device__ __forceinline__ void wait_hot()
    {
        if (!hot_n)
            return;
        if (!ag_sv_mbar_wait(&sh.mbar, mphase, p.mbar_spins)) {
            atomicOr(&p.ctl->fault, 1u);
            /* the copies may still be in flight: a long, bounded second chance */
            ag_sv_mbar_wait(&sh.mbar, mphase, 1u << 24);
        }
        mphase ^= 1u;
    }

    template <bool LOW> __device__ __forceinline__ float gather(uint32_t u) const
    {
        if (LOW)
            return ag_sv_low<PREC>(u < hot_n ? hot16[u] : ag_sv_ld_u16(c_in16 + u, pol_last, u < p.warm_n));
        return u < hot_n ? hot32[u] : ag_sv_ld_f32(c_in32 + u, pol_last, u < p.warm_n);
    }

    /* SpMV: the weights of a quad (quad k of q.ids) */
    __device__ __forceinline__ float4 weights(size_t k) const
    {
        if (p.wmode == AG_SPMV_W_GRAPH)
            return ag_ld_stream_f4(reinterpret_cast<const float4 *>(q.w) + k, pol_first);
        return p.wmode == AG_SPMV_W_CONST ? make_float4(0.0001f, 0.0001f, 0.0001f, 0.0001f)
                                          : make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    }

    __device__ __forceinline__ static void times(float4 &x, const float4 &w)
    {
        x.x = __fmul_rn(w.x, x.x);
        x.y = __fmul_rn(w.y, x.y);
        x.z = __fmul_rn(w.z, x.z);
        x.w = __fmul_rn(w.w, x.w);
    }

    /* the group gathers `n` slots (a multiple of 4 is staged) from slot k0 */
    template <bool LOW> __device__ __forceinline__ void stage(float *vals, uint64_t k0, uint32_t n) const
    {
        const uint4 *i4 = reinterpret_cast<const uint4 *>(q.ids + k0);
        const uint32_t n4 = (n + 3u) >> 2;
        for (uint32_t i = st; i < n4; i += 2u * AG_SUB_THREADS) {
            const bool two = i + AG_SUB_THREADS < n4;
            const uint4 a = ag_ld_stream_u4(i4 + i, pol_first);
            uint4 b = make_uint4(0, 0, 0, 0);
            if (two)
                b = ag_ld_stream_u4(i4 + i + AG_SUB_THREADS, pol_first);
            float4 x, y;
            x.x = gather<LOW>(a.x);
            x.y = gather<LOW>(a.y);
            x.z = gather<LOW>(a.z);
            x.w = gather<LOW>(a.w);
            y.x = gather<LOW>(b.x);
            y.y = gather<LOW>(b.y);
            y.z = gather<LOW>(b.z);
            y.w = gather<LOW>(b.w);
            if (MODE == AG_MODE_SPMV) {
                const float4 wx = weights((k0 >> 2) + i), wy = weights((k0 >> 2) + i + (two ? AG_SUB_THREADS : 0u));
                times(x, wx);
                times(y, wy);
            }
            reinterpret_cast<float4 *>(vals)[i] = x;
            if (two)
                reinterpret_cast<float4 *>(vals)[i + AG_SUB_THREADS] = y;
        }
    }

    /* ------------------------------------------------------------- update */
    __device__ __forceinline__ void put_c(uint32_t r, float c)
    {
        if (PREC != 0 && (flags & AG_GEN_WRITE_LOW))
            ag_st_keep_u16(c_out16 + r, ag_sv_to_low<PREC>(c), pol_last);
        else
            ag_st_keep_f32(c_out32 + r, c, pol_last);
    }

    /* the reference's per-vertex update for a finished row sum (rank at `at`,
     * device row r); data-driven
     * passes carry the row's tag in the sum's sign bit: rows off the worklist
     * and rows that moved by less than epsilon keep rank and contribution
     * (sign cleared, pageRank.c:2896-2916) */
    __device__ __forceinline__ void finish(uint32_t at, uint32_t r, float s, float rp, uint32_t od)
    {
        if (MODE == AG_MODE_SPMV) {
            /* a sum that starts at +0 never ends at -0 */
            q.y[p.perm ? __ldg(p.perm + r) : r] = __fadd_rn(s, 0.0f);
            return;
        }
        if (MODE == AG_MODE_DD) {
            if (iter == 0 || (__float_as_uint(s) >> 31)) {
                const float rn = __fadd_rn(p.base, __fmul_rn(p.damp, fabsf(s)));
                const double err = (double)fabsf(__fsub_rn(rn, rp));
                my_err += err;
                if (err >= eps) {
                    p.rank[at] = rn;
                    const float c = od ? __fdiv_rn(rn, __uint2float_rn(od)) : 0.0f;
                    ag_st_keep_f32(c_out32 + r, __uint_as_float(__float_as_uint(c) | 0x80000000u), pol_last);
                    ++my_active;
                    return;
                }
            }
            ag_st_keep_f32(c_out32 + r, fabsf(ag_sv_ld_f32(c_in32 + r, pol_last, false)), pol_last);
            return;
        }
        const float rn = __fadd_rn(p.base, __fmul_rn(p.damp, s));
        p.rank[at] = rn;
        const double err = (double)fabsf(__fsub_rn(rn, rp));
        my_err += err;
        my_active += (err >= eps) ? 1u : 0u;
        put_c(r, od ? __fdiv_rn(rn, __uint2float_rn(od)) : 0.0f);
    }

    /* data-driven: whether a sign is set among vals[0, n) */
    __device__ __forceinline__ static uint32_t signs(const float *vals, uint32_t n)
    {
        uint32_t x = 0;
        for (uint32_t j = 0; j < n; ++j)
            x |= __float_as_uint(vals[j]);
        return x;
    }

    /* ------------------------------------------------------------ row bin */
    template <bool LOW> __device__ __forceinline__ void row_bin(uint32_t k, float *vals)
    {
        const uint4 ha = __ldg(reinterpret_cast<const uint4 *>(q.bins + k));
        const uint4 hb = __ldg(reinterpret_cast<const uint4 *>(q.bins + k) + 1);
        const uint32_t r0 = ha.x, nrows = ha.y, ulong = (ha.z + 31u) >> 5, units = ulong + ((ha.w + 31u) >> 5);
        const uint32_t nslots = hb.x, gid = hb.y;
        if (MODE == AG_MODE_MULTI && (nrows == 0 || *((volatile uint32_t *)(p.g_done + gid))))
            return; /* the same for the whole group */
        const uint64_t k0 = (uint64_t)hb.z | ((uint64_t)hb.w << 32);
        const uint32_t lb = ag_bin_list(r0, k);
        float *sums = vals + ((nslots + 3u) & ~3u);
        /* what the sums and the update need first is on its way while the
         * gathers run */
        uint32_t e = 0, ub = 0, od = 0;
        float rp = 0.0f;
        if (sw < units) {
            e = __ldg(q.brow + lb + 32u * sw + lane);
            ub = __ldg(q.ubase + (lb >> 5) + sw);
        }
        if (MODE != AG_MODE_SPMV && st < nrows) {
            rp = ag_ld_rank(p.rank + r0 + st);
            od = ag_ld_row_u32(p.outdeg + r0 + st);
        }
        stage<LOW>(vals, k0, nslots);
        /* rows without in-edges sum to 0; a hub row is its composer's */
        if (nrows > ha.z + ha.w)
            for (uint32_t i = st; i < nrows; i += AG_SUB_THREADS) {
                float z = 0.0f;
                if (q.nhub && __ldg(p.row_off + r0 + i + 1) - __ldg(p.row_off + r0 + i) > AG_BIN_HUB)
                    z = __uint_as_float(AG_SV_HUB);
                sums[i] = z;
            }
        ag_sv_sub_sync(sub);
        for (uint32_t u = sw; u < units; u += AG_SUB_WARPS) {
            uint32_t en = 0, un = 0;
            if (u + AG_SUB_WARPS < units) {
                en = __ldg(q.brow + lb + 32u * (u + AG_SUB_WARPS) + lane);
                un = __ldg(q.ubase + (lb >> 5) + u + AG_SUB_WARPS);
            }
            const uint32_t len = e >> 16;
            if (u < ulong) {
                /* 32 long rows, one after another in the buffer */
                const uint32_t pad = (len + 3u) & ~3u;
                uint32_t at = pad;
#pragma unroll
                for (uint32_t o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(0xffffffffu, at, o);
                    if (lane >= o)
                        at += t;
                }
                at += ub - pad;
                if (len) {
                    uint32_t tag = 0;
                    float s = EXACT ? ag_sv_chain<MODE>(vals + at, len, -0.0f) : ag_sv_fast<MODE>(vals + at, len, tag);
                    if (MODE == AG_MODE_DD && EXACT)
                        tag = signs(vals + at, len);
                    if (MODE == AG_MODE_DD)
                        s = __uint_as_float(__float_as_uint(s) | (tag & 0x80000000u));
                    sums[e & 0xffffu] = s;
                }
            } else {
                const float *v = vals + ub + lane;
                const uint32_t most = __shfl_sync(0xffffffffu, len, 0); /* longest first */
                float s = -0.0f; /* -0 + x = x */
                uint32_t neg = 0;
                for (uint32_t i = 0; i < most; i += 4) {
                    float x[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        x[t] = i + t < len ? v[32u * (i + t)] : MODE == AG_MODE_DD ? 0.0f : -0.0f;
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        if (MODE == AG_MODE_DD) {
                            neg |= __float_as_uint(x[t]); /* (s's own sign goes) */
                            x[t] = fabsf(x[t]);
                        }
                        s = __fadd_rn(s, x[t]); /* s + -0 = s */
                    }
                }
                if (MODE == AG_MODE_DD)
                    s = __uint_as_float((__float_as_uint(s) & 0x7fffffffu) | (neg & 0x80000000u));
                if (len)
                    sums[e & 0xffffu] = s;
            }
            e = en;
            ub = un;
        }
        ag_sv_sub_sync(sub);
        for (uint32_t i = st; i < nrows; i += AG_SUB_THREADS) {
            float rn = 0.0f;
            uint32_t on = 0;
            if (MODE != AG_MODE_SPMV && i + AG_SUB_THREADS < nrows) {
                rn = ag_ld_rank(p.rank + r0 + i + AG_SUB_THREADS);
                on = ag_ld_row_u32(p.outdeg + r0 + i + AG_SUB_THREADS);
            }
            const float s = sums[i];
            if (__float_as_uint(s) != AG_SV_HUB ||
                __ldg(p.row_off + r0 + i + 1) - __ldg(p.row_off + r0 + i) <= AG_BIN_HUB)
                finish(r0 + i, r0 + i, s, rp, od);
            rp = rn;
            od = on;
        }
        if (MODE == AG_MODE_MULTI)
            graph_totals(gid);
        ag_sv_sub_sync(sub);
    }

    /* this thread's totals go to a graph of the union */
    __device__ __forceinline__ void graph_totals(uint32_t gid)
    {
        const double e = ag_sv_warp_d(my_err);
        const uint32_t a = __reduce_add_sync(0xffffffffu, my_active);
        if (lane == 0) {
            if (e != 0.0)
                atomicAdd(p.g_err + gid, e);
            if (a)
                atomicAdd(p.g_active + gid, a);
        }
        my_err = 0.0;
        my_active = 0;
    }

    __device__ __forceinline__ uint32_t graph_of(uint32_t r) const
    {
        uint32_t lo = 0, hi = p.ngraphs;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(p.gstart + mid) <= r)
                lo = mid;
            else
                hi = mid;
        }
        return lo;
    }

    /* maps of a round from its values (eight per lane).  A round that should
     * leave its binade (it did in the pass before) keeps the lanes' maps and
     * values for the composer. */
    __device__ __forceinline__ void map_round(const float *v, uint32_t pred, uint32_t next, uint4 *words)
    {
        const uint32_t lo = ag_sv_low_exp(pred, next);
        uint32_t w0 = AG_XNOT, w1 = AG_XNOT, slot = AG_SV_NOT_KEPT;
        if (lo >= 24u && lo < 254u) {
            uint32_t a0, a1, b0, b1;
            ag_sv_moves(v, lo, a0, a1);
            ag_sv_moves(v, lo + 1u, b0, b1);
            if ((next >> 7) > (pred >> 7)) {
                if (lane == 0)
                    slot = atomicAdd(q.sync + AG_SYNC_KEPT, 1u);
                slot = __shfl_sync(0xffffffffu, slot, 0);
                if (slot < q.kept_cap) {
                    float4 *k = q.kept + (size_t)slot * AG_KEPT_QUADS;
                    reinterpret_cast<uint4 *>(k)[lane] = make_uint4(a0, a1, b0, b1);
                    k[32 + 2 * lane] = make_float4(v[0], v[1], v[2], v[3]);
                    k[33 + 2 * lane] = make_float4(v[4], v[5], v[6], v[7]);
                } else {
                    slot = AG_SV_NOT_KEPT;
                }
            }
            ag_sv_scan(lane, a0, a1);
            ag_sv_scan(lane, b0, b1);
            w0 = ag_sv_pack(a0, a1);
            w1 = ag_sv_pack(b0, b1);
        }
        if (lane == 31)
            *words = make_uint4(w0, w1, slot, 0u);
    }

    /* ------------------------------------------------------------ hub bin */
    /* Chunks [c0, c0 + nc) of hub rows, staged together.  FAST: a warp sums
     * each chunk.  EXACT: the rounds of 256 values of a chunk are mapped by
     * any warps, each at the exponent where the round began in the pass
     * before; a row's first AG_BIN_HEAD values are one lane's chain.  The last
     * chunk of a row to arrive composes the row. */
    template <bool LOW> __device__ __forceinline__ void hub_bin(uint32_t k, float *vals)
    {
        const uint32_t c0 = k * q.per_bin, nc = min(q.per_bin, q.nhub - c0);
        if (EXACT)
            for (uint32_t i = st; i <= nc * AG_BIN_ROUNDS; i += AG_SUB_THREADS)
                sh.pred[sub][i] = __ldcg(q.hub_pred + (size_t)c0 * AG_BIN_ROUNDS + i);
        stage<LOW>(vals, (uint64_t)c0 * AG_BIN_HUB, nc * AG_BIN_HUB);
        ag_sv_sub_sync(sub);
        if (EXACT) {
            for (uint32_t t = sw; t < nc * AG_BIN_ROUNDS; t += AG_SUB_WARPS) {
                const uint32_t ch = t / AG_BIN_ROUNDS, rd = t % AG_BIN_ROUNDS;
                const uint4 h = __ldg(q.hubs + c0 + ch);
                const uint32_t len = (h.w & (AG_BIN_HUB - 1u)) + 1u;
                const float *v0 = vals + ch * AG_BIN_HUB;
                if (h.y == 0 && rd < AG_BIN_HEAD / AG_BIN_ROUND) {
                    if (rd == 0 && lane == 0)
                        q.hub_sum[c0 + ch] = (double)ag_sv_chain<MODE>(v0, AG_BIN_HEAD, -0.0f);
                    continue;
                }
                if (rd * AG_BIN_ROUND >= len)
                    continue;
                float v[8];
                ag_sv_eight<MODE>(v0 + rd * AG_BIN_ROUND, len - rd * AG_BIN_ROUND, lane, v);
                const size_t k = (size_t)c0 * AG_BIN_ROUNDS + t;
                map_round(v, sh.pred[sub][t], sh.pred[sub][t + 1], q.hub_words + k);
            }
            ag_sv_sub_sync(sub);
        }
        for (uint32_t ch = sw; ch < nc; ch += AG_SUB_WARPS) {
            const uint4 h = __ldg(q.hubs + c0 + ch);
            const uint32_t len = (h.w & (AG_BIN_HUB - 1u)) + 1u, nch = h.w >> 11;
            float *v0 = vals + ch * AG_BIN_HUB;
            uint32_t tag = 0;
            if (MODE == AG_MODE_DD && EXACT)
                for (uint32_t j = lane; j < len; j += 32)
                    tag |= __float_as_uint(v0[j]);
            if (!EXACT) {
                double t = 0.0;
                for (uint32_t j = lane; j < len; j += 256) {
                    float x[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        x[i] = j + 32u * i < len ? v0[j + 32u * i] : 0.0f;
                        if (MODE == AG_MODE_DD) {
                            tag |= __float_as_uint(x[i]);
                            x[i] = fabsf(x[i]);
                        }
                    }
                    t += (double)__fadd_rn(__fadd_rn(__fadd_rn(x[0], x[1]), __fadd_rn(x[2], x[3])),
                                           __fadd_rn(__fadd_rn(x[4], x[5]), __fadd_rn(x[6], x[7])));
                }
                t = ag_sv_warp_d(t);
                if (lane == 0)
                    q.hub_sum[c0 + ch] = t;
            }
            /* the chunk's tag: a bit of the row's arrival word */
            if (MODE == AG_MODE_DD && __any_sync(0xffffffffu, tag >> 31) && lane == 0)
                atomicOr(q.hub_seen + h.z, 0x80000000u);
            uint32_t seen = 0;
            __syncwarp();
            if (lane == 0) {
                __threadfence();
                seen = atomicAdd(q.hub_seen + h.z, 1u);
            }
            seen = __shfl_sync(0xffffffffu, seen, 0);
            if ((seen & 0x7fffffffu) != nch - 1u)
                continue;
            __threadfence();
            float s;
            if (EXACT) {
                s = compose<LOW>(h);
            } else {
                double t = 0.0;
                for (uint32_t c = lane; c < nch; c += 32)
                    t += __ldcg(q.hub_sum + h.z + c);
                s = __double2float_rn(ag_sv_warp_d(t));
            }
            if (lane == 0) {
                if (MODE == AG_MODE_DD && (seen >> 31 || (*((volatile uint32_t *)(q.hub_seen + h.z)) >> 31)))
                    s = __uint_as_float(__float_as_uint(s) | 0x80000000u);
                q.hub_seen[h.z] = 0;
                const uint32_t r = h.x;
                if (MODE != AG_MODE_MULTI || !*((volatile uint32_t *)(p.g_done + graph_of(r))))
                    finish(r, r, s, MODE == AG_MODE_SPMV ? 0.0f : ag_ld_rank(p.rank + r), ag_ld_row_u32(p.outdeg + r));
            }
            __syncwarp();
            if (MODE == AG_MODE_MULTI)
                graph_totals(graph_of(h.x));
        }
        ag_sv_sub_sync(sub);
    }

    /* EXACT order: a hub row on one warp, its rounds in order from its head
     * sum, 32 at a time.  Maps at s's exponent compose (a scan of the lanes'
     * maps); the first that does not apply is added from its values
     * (ag_sv_round), kept by the chunk or gathered again, and the rounds after
     * it go on.  Records where each round began. */
    template <bool LOW> __device__ float compose(const uint4 h)
    {
        const uint32_t deg = __ldg(p.row_off + h.x + 1) - __ldg(p.row_off + h.x);
        const uint32_t rounds = (deg + AG_BIN_ROUND - 1u) / AG_BIN_ROUND;
        const size_t k0 = (size_t)h.z * AG_BIN_ROUNDS;
        const uint4 *words = q.hub_words + k0;
        uint16_t *pred = q.hub_pred + k0;
        float s = (float)__ldcg(q.hub_sum + h.z);
        bool below = false; /* SpMV: the last round added by its values had one below zero */
        uint4 wn = make_uint4(0, 0, 0, 0);
        uint32_t en = 0, em = 0;
        if (lane < rounds) {
            wn = __ldcg(words + lane);
            en = __ldcg(pred + lane);
            em = __ldcg(pred + lane + 1);
        }
        for (uint32_t b = 0; b < rounds; b += 32) {
            const uint4 w = wn;
            const uint32_t lo = ag_sv_low_exp(en, em), k = b + lane;
            uint32_t began = en;
            if (k + 32u < rounds) {
                wn = __ldcg(words + k + 32u);
                en = __ldcg(pred + k + 32u);
                em = __ldcg(pred + k + 33u);
            }
            const bool live = k < rounds && k >= AG_BIN_HEAD / AG_BIN_ROUND;
            uint32_t done = b ? 0u : AG_BIN_HEAD / AG_BIN_ROUND;
            /* rounds without a map at all */
            uint32_t none = 0;
            if (MODE == AG_MODE_SPMV)
                none = __ballot_sync(0xffffffffu, live && (w.x & w.y & AG_XNOT) && w.z == AG_SV_NOT_KEPT);
            while (done < 32u && b + done < rounds) {
                const uint32_t sb = __float_as_uint(s), ex = sb >> 23;
                const uint32_t m = (sb & 0x7fffffu) | 0x800000u;
                uint32_t d0 = 0, d1 = 0;
                if (live && lane >= done) {
                    const uint32_t x = ex == lo ? w.x : ex == lo + 1u ? w.y : AG_XNOT;
                    if ((x & AG_XNOT) || ex < 24u || ex > 254u) {
                        d0 = d1 = 1u << 24;
                    } else {
                        d0 = x & 0x3ffffffu;
                        d1 = d0 + ((x >> 26) & 3u) - 1u;
                    }
                }
                uint32_t ok = ~(1u << done);
                uint32_t to = 0;
                if (MODE != AG_MODE_SPMV || !((none >> done) & 1u)) {
                    ag_sv_scan(lane, d0, d1);
                    to = m + ((m & 1u) ? d1 : d0);
                    ok = __ballot_sync(0xffffffffu, to < (1u << 24));
                }
                const uint32_t out = ok == 0xffffffffu ? 32u : __ffs(~ok) - 1;
                const uint32_t before = __shfl_sync(0xffffffffu, to, (out - 1u) & 31u);
                const uint32_t prev = __shfl_up_sync(0xffffffffu, to, 1);
                if (lane >= done && lane <= out)
                    began = (ex << 7) | (((lane > done ? prev : m) >> 16) & 0x7fu);
                if (out > done)
                    s = ag_sv_make(ex, before);
                done = out;
                if (out == 32u)
                    break;
                /* this round from its values, eight consecutive ones per lane */
                const uint32_t r = b + out, slot = __shfl_sync(0xffffffffu, w.z, out);
                if (MODE == AG_MODE_SPMV && below && out < 31u && ((none >> out) & 3u) == 3u) {
                    /* two such rounds, 16 consecutive values per lane: half
                     * the hand-overs of s from lane to lane */
                    const size_t kq = (k0 + r) * (AG_BIN_ROUND / 4) + 4u * lane;
                    const uint4 *src = reinterpret_cast<const uint4 *>(q.ids) + kq;
                    const uint32_t j = r * AG_BIN_ROUND + 16u * lane;
                    if (j + 2u * AG_BIN_ROUND < deg) {
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(src + AG_BIN_ROUND / 2));
                        if (p.wmode == AG_SPMV_W_GRAPH)
                            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const float4 *>(q.w) + kq +
                                                                         AG_BIN_ROUND / 2));
                    }
                    float v[16];
                    gather8<LOW>(__ldg(src), __ldg(src + 1), j, deg, kq, kq + 1, v);
                    gather8<LOW>(__ldg(src + 2), __ldg(src + 3), j + 8u, deg, kq + 2, kq + 3, v + 8);
                    s = ag_sv_serial<16>(v, s, 0u);
                    done = out + 2u;
                    continue;
                }
                const uint32_t e0 = __shfl_sync(0xffffffffu, lo, out);
                float v[8];
                uint32_t from = 0;
                if (slot != AG_SV_NOT_KEPT) {
                    const float4 *kp = q.kept + (size_t)slot * AG_KEPT_QUADS;
                    const uint4 mp = __ldcg(reinterpret_cast<const uint4 *>(kp) + lane);
                    const float4 x = __ldcg(kp + 32 + 2 * lane), y = __ldcg(kp + 33 + 2 * lane);
                    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
                    v[4] = y.x, v[5] = y.y, v[6] = y.z, v[7] = y.w;
                    if ((__float_as_uint(s) >> 23) == e0) {
                        /* the lanes' maps below the binade's end, the lane that
                         * leaves it value by value, the others' maps above it */
                        from = mapped(mp.x, mp.y, v, 0u, s);
                        if (from < 32u && (__float_as_uint(s) >> 23) == e0 + 1u)
                            from = mapped(mp.z, mp.w, v, from, s);
                    }
                } else {
                    const size_t kq = (k0 + r) * (AG_BIN_ROUND / 4) + 2u * lane;
                    const uint4 *src = reinterpret_cast<const uint4 *>(q.ids) + kq;
                    const uint32_t later = out < 31u ? none >> (out + 1u) : 0u;
                    if (MODE == AG_MODE_SPMV && later) {
                        /* the next of these rounds */
                        const uint32_t d = __ffs(later) * (AG_BIN_ROUND / 4);
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(src + d));
                        if (p.wmode == AG_SPMV_W_GRAPH)
                            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const float4 *>(q.w) + kq + d));
                    }
                    gather8<LOW>(__ldg(src), __ldg(src + 1), r * AG_BIN_ROUND + 8u * lane, deg, kq, kq + 1, v);
                    if (MODE == AG_MODE_DD)
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            v[i] = fabsf(v[i]);
                }
                /* SpMV: a value below zero moves M back, so no map holds and the
                 * round is added value by value.  us per product, EXACT, weighted
                 * R-MAT, the three launches / rounds one by one / here, x centred
                 * on 0: 1 M vertices 443 / 421 / 338, 4 M 1115 / 1217 / 1010; one
                 * x in 1000 below zero: 283 / 240 / 222, 745 / 857 / 780 */
                if (MODE == AG_MODE_SPMV) {
                    bool bad = false;
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        bad |= !(v[i] >= 0.0f);
                    below = __any_sync(0xffffffffu, bad);
                    if (below) {
                        s = ag_sv_serial<8>(v, s, from);
                        from = 32u;
                    }
                }
                if (from < 32u)
                    s = ag_sv_round(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], s, lane, from);
                done = out + 1u;
            }
            if (live)
                pred[k] = (uint16_t)min(began, 0x7fffu);
        }
        return s;
    }

    /* lanes from `done` on move s by their maps (at s's exponent); the lane
     * where s would leave its binade adds its values v.  Returns the lanes
     * that are in s. */
    __device__ __forceinline__ uint32_t mapped(uint32_t d0, uint32_t d1, const float *v, uint32_t done, float &s) const
    {
        const uint32_t sb = __float_as_uint(s), ex = sb >> 23, m = (sb & 0x7fffffu) | 0x800000u;
        if (lane < done)
            d0 = d1 = 0;
        ag_sv_scan(lane, d0, d1);
        const uint32_t to = m + ((m & 1u) ? d1 : d0);
        const uint32_t ok = __ballot_sync(0xffffffffu, to < (1u << 24));
        if (ok == 0xffffffffu) {
            s = ag_sv_make(ex, __shfl_sync(0xffffffffu, to, 31));
            return 32u;
        }
        const uint32_t out = __ffs(~ok) - 1;
        const uint32_t before = __shfl_sync(0xffffffffu, to, (out - 1u) & 31u);
        s = ag_sv_make(ex, out ? before : m);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            s = __fadd_rn(s, v[i]);
        s = __shfl_sync(0xffffffffu, s, out);
        return out + 1u;
    }

    /* EXACT order, before the first pass: each round's starting exponent from
     * plain sums of the first contributions, so that the first pass composes
     * like the later ones (added value by value it took 2 to 6 ms at R-MAT
     * scale 22 to 24, 6 to 15 later passes).  Two grid barriers. */
    template <bool LOW> __device__ __forceinline__ bool predict(float *vals)
    {
        for (uint32_t k = blockIdx.x + sub * gridDim.x; k < q.nhb; k += gridDim.x * AG_SUBS) {
            const uint32_t c0 = k * q.per_bin, nc = min(q.per_bin, q.nhub - c0);
            stage<LOW>(vals, (uint64_t)c0 * AG_BIN_HUB, nc * AG_BIN_HUB);
            ag_sv_sub_sync(sub);
            for (uint32_t t = sw; t < nc * AG_BIN_ROUNDS; t += AG_SUB_WARPS) {
                const uint4 h = __ldg(q.hubs + c0 + t / AG_BIN_ROUNDS);
                const uint32_t len = (h.w & (AG_BIN_HUB - 1u)) + 1u, rd = t % AG_BIN_ROUNDS;
                float x = 0.0f;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint32_t j = rd * AG_BIN_ROUND + lane + 32u * i;
                    if (j < len)
                        x += fabsf(vals[(t / AG_BIN_ROUNDS) * AG_BIN_HUB + j]);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                    x += __shfl_xor_sync(0xffffffffu, x, o);
                if (lane == 0)
                    q.hub_words[(size_t)c0 * AG_BIN_ROUNDS + t].x = __float_as_uint(x);
            }
            ag_sv_sub_sync(sub);
        }
        return predict_scan();
    }

    __device__ __forceinline__ bool predict_scan()
    {
        const uint32_t f = flags;
        if (!grid_sync([&] { return f; }))
            return false;
        const uint32_t nw = gridDim.x * (AG_SOLVE_BLK / 32);
        for (uint32_t c = blockIdx.x * (AG_SOLVE_BLK / 32) + (tid >> 5); c < q.nhub; c += nw) {
            const uint4 h = __ldg(q.hubs + c);
            if (h.y != 0)
                continue;
            const uint32_t total = (h.w >> 11) * AG_BIN_ROUNDS;
            float run = 0.0f;
            for (uint32_t b = 0; b < total; b += 32) {
                const uint32_t k = b + lane;
                const float x =
                    k < total ? __uint_as_float(__ldcg(&q.hub_words[(size_t)c * AG_BIN_ROUNDS + k].x)) : 0.0f;
                float inc = x;
#pragma unroll
                for (uint32_t o = 1; o < 32; o <<= 1) {
                    const float t = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o)
                        inc += t;
                }
                if (k < total)
                    q.hub_pred[(size_t)c * AG_BIN_ROUNDS + k] =
                        (uint16_t)(__float_as_uint(run + (inc - x)) >> 16);
                run += __shfl_sync(0xffffffffu, inc, 31);
            }
        }
        return grid_sync([&] { return f; });
    }

    /* -------------------------------------------------------------- units */
    /* eight gathered values of a lane's two quads (quads ka and kb of q.ids);
     * those at or past n are -0 (s + -0 = s) */
    template <bool LOW> __device__ __forceinline__ void gather8(const uint4 &a, const uint4 &b, uint32_t j, uint32_t n, size_t ka, size_t kb,
                                            float *v) const
    {
        float4 x, y, wx = make_float4(0.0f, 0.0f, 0.0f, 0.0f), wy = wx;
        if (MODE == AG_MODE_SPMV) {
            if (j < n)
                wx = weights(ka);
            if (j + 4u < n)
                wy = weights(kb);
        }
        x.x = gather<LOW>(a.x);
        x.y = gather<LOW>(a.y);
        x.z = gather<LOW>(a.z);
        x.w = gather<LOW>(a.w);
        y.x = gather<LOW>(b.x);
        y.y = gather<LOW>(b.y);
        y.z = gather<LOW>(b.z);
        y.w = gather<LOW>(b.w);
        if (MODE == AG_MODE_SPMV) {
            times(x, wx);
            times(y, wy);
        }
        v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
        v[4] = y.x, v[5] = y.y, v[6] = y.z, v[7] = y.w;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (j + i >= n)
                v[i] = -0.0f;
    }

    /* a lane's running sum over eight more values of its row of n in-edges */
    struct RowSum
    {
        float s;      /* stream order                                          */
        double t;     /* FAST order, rows above AG_BIN_SEQ in-edges            */
        uint32_t neg; /* data-driven: sign bits                                */
    };

    __device__ __forceinline__ void add8(RowSum &a, float *v, uint32_t n) const
    {
        if (MODE == AG_MODE_DD) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                /* -0 past the end is no tag: its other bits are 0 */
                a.neg |= v[i] != 0.0f ? __float_as_uint(v[i]) : 0u;
                v[i] = fabsf(v[i]);
            }
        }
        if (!EXACT && n > AG_BIN_SEQ) {
            a.t += (double)__fadd_rn(__fadd_rn(__fadd_rn(v[0], v[1]), __fadd_rn(v[2], v[3])),
                                     __fadd_rn(__fadd_rn(v[4], v[5]), __fadd_rn(v[6], v[7])));
            return;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            a.s = __fadd_rn(a.s, v[i]);
    }

    __device__ __forceinline__ void unit_finish(uint32_t u, uint32_t info, const RowSum &sum, float rp, uint32_t od)
    {
        const uint32_t at = 32u * u + lane, n = AG_UNIT_LEN(info);
        if (at >= p.N || (info & AG_UNIT_HUB))
            return;
        float s = n ? sum.s : 0.0f;
        if (!EXACT && n > AG_BIN_SEQ)
            s = __double2float_rn(sum.t);
        if (MODE == AG_MODE_DD)
            s = __uint_as_float((__float_as_uint(s) & 0x7fffffffu) | (sum.neg & 0x80000000u));
        finish(at, (at & ~(AG_UNIT_WIN - 1u)) + AG_UNIT_ROW(info), s, rp, od);
    }

    /* the units with the longest rows, one after another */
    template <bool LOW> __device__ __forceinline__ void heavy_unit(uint32_t u)
    {
        const uint32_t b0 = __ldg(q.ubaseq + u), rounds = (__ldg(q.ubaseq + u + 1) - b0) >> 5;
        uint32_t info = 0, od = 0;
        float rp = 0.0f;
        unit_row(u, info, rp, od);
        const uint32_t n = AG_UNIT_LEN(info);
        uint4 a = make_uint4(0, 0, 0, 0), b = a;
        pair(b0, rounds, a, b);
        RowSum sum = {-0.0f, 0.0, 0u};
        for (uint32_t i = 0; i < rounds; i += 2) {
            uint4 na = make_uint4(0, 0, 0, 0), nb = na;
            if (i + 2 < rounds)
                pair(b0 + 32u * (i + 2), rounds - i - 2, na, nb);
            float v[8];
            gather8<LOW>(a, b, 4u * i, n, unit_quad(b0, i), unit_quad(b0, i + 1), v);
            add8(sum, v, n);
            a = na;
            b = nb;
        }
        unit_finish(u, info, sum, rp, od);
    }

    /* the other units, a batch of consecutive ones at a time from an atomic
     * counter (batch bt first, then those of the tickets drawn, first_ticket
     * added modulo 2^32).  The next quads (of this unit or the next one) are on their way
     * while a lane's eight gathers travel, and the next batch is drawn one
     * batch ahead. */
    template <bool LOW> __device__ __forceinline__ void units(uint32_t bt, uint32_t first_ticket)
    {
        if (bt >= q.nbatch)
            return;
        uint32_t u = __ldg(q.bstart + bt), end = __ldg(q.bstart + bt + 1);
        uint32_t un = u, unn;         /* the next unit, the one after it */
        uint32_t start_n = 0, end_n = 0;
        uint32_t ticket = 0; /* lane 0: of the batch after the next one */
        auto draw = [&]() {
            bt = __shfl_sync(0xffffffffu, ticket, 0) + first_ticket;
            start_n = end_n = q.nunits;
            if (bt < q.nbatch) {
                start_n = __ldg(q.bstart + bt);
                end_n = __ldg(q.bstart + bt + 1);
                if (lane == 0)
                    ticket = atomicAdd(q.sync + AG_SYNC_BIN, 1u);
            }
        };
        /* the unit after x in this warp's batches */
        auto after = [&](uint32_t x) {
            ++x;
            while (x >= end && x < q.nunits) {
                x = start_n;
                end = end_n;
                draw();
            }
            return x;
        };
        if (lane == 0)
            ticket = atomicAdd(q.sync + AG_SYNC_BIN, 1u);
        draw();
        if (u >= end) /* an empty batch */
            u = after(u - 1u);
        if (u >= q.nunits)
            return;
        un = after(u);
        uint32_t b0, rounds, info = 0, od = 0, bn, rn;
        float rp = 0.0f;
        unit_base(u, b0, rounds);
        unit_base(un, bn, rn);
        unit_row(u, info, rp, od);
        uint4 a = make_uint4(0, 0, 0, 0), b = a;
        pair(b0, rounds <= q.heavy_quads ? rounds : 0u, a, b);
        for (;;) {
            uint32_t info_n = 0, od_n = 0, bnn = 0, rnn = 0;
            float rp_n = 0.0f;
            unn = un;
            if (un < q.nunits) {
                unit_row(un, info_n, rp_n, od_n);
                unn = after(un); /* q.nunits once they are used up */
                unit_base(unn, bnn, rnn);
            }
            const uint32_t n = AG_UNIT_LEN(info), first_n = rn <= q.heavy_quads ? rn : 0u;
            if (rounds <= q.heavy_quads) {
                RowSum sum = {-0.0f, 0.0, 0u};
                for (uint32_t i = 0; i < rounds; i += 2) {
                    uint4 na = make_uint4(0, 0, 0, 0), nb = na;
                    if (i + 2 < rounds)
                        pair(b0 + 32u * (i + 2), rounds - i - 2, na, nb);
                    else
                        pair(bn, first_n, na, nb);
                    float v[8];
                    gather8<LOW>(a, b, 4u * i, n, unit_quad(b0, i), unit_quad(b0, i + 1), v);
                    add8(sum, v, n);
                    a = na;
                    b = nb;
                }
                unit_finish(u, info, sum, rp, od);
            }
            if (rounds == 0 || rounds > q.heavy_quads)
                pair(bn, first_n, a, b);
            if (un >= q.nunits)
                return;
            u = un;
            b0 = bn;
            rounds = rn;
            un = unn;
            bn = bnn;
            rn = rnn;
            info = info_n;
            rp = rp_n;
            od = od_n;
        }
    }

    __device__ __forceinline__ void unit_base(uint32_t u, uint32_t &b0, uint32_t &rounds) const
    {
        b0 = rounds = 0;
        if (u < q.nunits) {
            b0 = __ldg(q.ubaseq + u);
            rounds = (__ldg(q.ubaseq + u + 1) - b0) >> 5;
        }
    }

    __device__ __forceinline__ void unit_row(uint32_t u, uint32_t &info, float &rp, uint32_t &od) const
    {
        const uint32_t at = 32u * u + lane;
        if (at < p.N) {
            info = ag_ld_row_u32(q.info + at);
            if (MODE != AG_MODE_SPMV) {
                rp = ag_ld_rank(p.rank + at);
                od = ag_ld_row_u32(q.uoutdeg + at);
            }
        }
    }

    /* quad i of this lane's row in a unit, as a quad of q.ids */
    __device__ __forceinline__ size_t unit_quad(uint32_t b0, uint32_t i) const
    {
        return (size_t)q.nhub * (AG_BIN_HUB / 4) + b0 + 32u * i + lane;
    }

    /* this lane's quads at b0 and b0 + 32, as far as `left` rounds go */
    __device__ __forceinline__ void pair(uint32_t b0, uint32_t left, uint4 &a, uint4 &b) const
    {
        if (left > 0)
            a = ag_ld_stream_u4(q.uids + b0 + lane, pol_first);
        if (left > 1)
            b = ag_ld_stream_u4(q.uids + b0 + 32u + lane, pol_first);
    }

    /* EXACT order: the first AG_BIN_HEAD values of 32 hub rows, one row per lane */
    template <bool LOW> __device__ __forceinline__ void heads(uint32_t k)
    {
        const uint32_t i = 32u * k + lane;
        if (i >= q.nhrow)
            return;
        const uint32_t first = __ldg(q.hrow + i);
        const uint4 *src = reinterpret_cast<const uint4 *>(q.ids) + (size_t)first * (AG_BIN_HUB / 4);
        RowSum sum = {-0.0f, 0.0, 0u};
        uint4 a = ag_ld_stream_u4(src, pol_first), b = ag_ld_stream_u4(src + 1, pol_first);
        for (uint32_t j = 0; j < AG_BIN_HEAD; j += 8) {
            uint4 na = a, nb = b;
            if (j + 8 < AG_BIN_HEAD) {
                na = ag_ld_stream_u4(src + j / 4 + 2, pol_first);
                nb = ag_ld_stream_u4(src + j / 4 + 3, pol_first);
            }
            float v[8];
            gather8<LOW>(a, b, j, AG_BIN_HEAD, (size_t)first * (AG_BIN_HUB / 4) + j / 4,
                    (size_t)first * (AG_BIN_HUB / 4) + j / 4 + 1, v);
            add8(sum, v, 0);
            a = na;
            b = nb;
        }
        q.hub_sum[first] = (double)sum.s;
        if (MODE == AG_MODE_DD)
            q.hub_tag[first] = sum.neg >> 31;
    }

    /* a hub chunk on one warp, a lane's eight values of a round in registers;
     * FAST: its sum; EXACT: its rounds' maps (predict: their plain sums) */
    template <bool PREDICT, bool LOW> __device__ __forceinline__ void chunk(uint32_t c)
    {
        const uint4 h = __ldg(q.hubs + c);
        const uint32_t len = (h.w & (AG_BIN_HUB - 1u)) + 1u;
        const uint32_t rounds = (len + AG_BIN_ROUND - 1u) / AG_BIN_ROUND;
        const bool head = EXACT && !PREDICT && h.y == 0;
        const uint4 *src = reinterpret_cast<const uint4 *>(q.ids) + (size_t)c * (AG_BIN_HUB / 4) + 2u * lane;
        uint32_t rd = head ? AG_BIN_HEAD / AG_BIN_ROUND : 0u;
        uint32_t pred = 0, next = 0;
        if (EXACT && !PREDICT && rd < rounds) {
            pred = __ldcg(q.hub_pred + (size_t)c * AG_BIN_ROUNDS + rd);
            next = __ldcg(q.hub_pred + (size_t)c * AG_BIN_ROUNDS + rd + 1);
        }
        uint4 a = make_uint4(0, 0, 0, 0), b = a;
        if (rd < rounds) {
            a = ag_ld_stream_u4(src + rd * (AG_BIN_ROUND / 4), pol_first);
            b = ag_ld_stream_u4(src + rd * (AG_BIN_ROUND / 4) + 1, pol_first);
        }
        double t = 0.0;
        uint32_t neg = 0;
        for (; rd < rounds; ++rd) {
            uint4 na = a, nb = b;
            uint32_t after = 0;
            if (EXACT && !PREDICT)
                after = __ldcg(q.hub_pred + (size_t)c * AG_BIN_ROUNDS + rd + 2);
            if (rd + 1 < rounds) {
                na = ag_ld_stream_u4(src + (rd + 1) * (AG_BIN_ROUND / 4), pol_first);
                nb = ag_ld_stream_u4(src + (rd + 1) * (AG_BIN_ROUND / 4) + 1, pol_first);
            }
            float v[8];
            const size_t kq = (size_t)c * (AG_BIN_HUB / 4) + rd * (AG_BIN_ROUND / 4) + 2u * lane;
            gather8<LOW>(a, b, rd * AG_BIN_ROUND + 8u * lane, len, kq, kq + 1, v);
            if (MODE == AG_MODE_DD) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    neg |= v[i] != 0.0f ? __float_as_uint(v[i]) : 0u;
                    v[i] = fabsf(v[i]);
                }
            }
            if (PREDICT) {
                float x = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                    x += __shfl_xor_sync(0xffffffffu, x, o);
                if (lane == 0)
                    q.hub_words[(size_t)c * AG_BIN_ROUNDS + rd].x = __float_as_uint(x);
            } else if (EXACT) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    v[i] = __fadd_rn(v[i], 0.0f); /* past the end: +0 */
                const size_t k = (size_t)c * AG_BIN_ROUNDS + rd;
                map_round(v, pred, next, q.hub_words + k);
                pred = next;
                next = after;
            } else {
                t += (double)__fadd_rn(__fadd_rn(__fadd_rn(v[0], v[1]), __fadd_rn(v[2], v[3])),
                                       __fadd_rn(__fadd_rn(v[4], v[5]), __fadd_rn(v[6], v[7])));
            }
            a = na;
            b = nb;
        }
        if (PREDICT) {
            if (lane >= rounds && lane < AG_BIN_ROUNDS)
                q.hub_words[(size_t)c * AG_BIN_ROUNDS + lane].x = 0u;
            return;
        }
        if (!EXACT) {
            t = ag_sv_warp_d(t);
            if (lane == 0)
                q.hub_sum[c] = t;
        }
        if (MODE == AG_MODE_DD) {
            neg = __any_sync(0xffffffffu, neg >> 31) ? 1u : 0u;
            /* a row's first chunk shares its tag with its head */
            if (lane == 0)
                q.hub_tag[head ? q.nhub + c : c] = neg;
        }
    }

    /* the hub rows from their chunks, a warp each (a grid barrier before it) */
    template <bool LOW> __device__ __forceinline__ void hub_rows()
    {
        for (uint32_t i = (tid >> 5) * gridDim.x + blockIdx.x; i < q.nhrow; i += gridDim.x * (AG_SOLVE_BLK / 32)) {
            const uint4 h = __ldg(q.hubs + __ldg(q.hrow + i));
            const uint32_t at = __ldg(q.posof + h.x), nch = h.w >> 11;
            float rp = 0.0f;
            uint32_t od = 0, tag = 0;
            if (MODE != AG_MODE_SPMV && lane == 0) {
                rp = ag_ld_rank(p.rank + at);
                od = ag_ld_row_u32(q.uoutdeg + at);
            }
            if (MODE == AG_MODE_DD) {
                for (uint32_t c = lane; c < nch; c += 32)
                    tag |= __ldcg(q.hub_tag + h.z + c);
                if (EXACT)
                    tag |= __ldcg(q.hub_tag + q.nhub + h.z);
            }
            float s;
            if (EXACT) {
                s = compose<LOW>(h);
            } else {
                double t = 0.0;
                for (uint32_t c = lane; c < nch; c += 32)
                    t += __ldcg(q.hub_sum + h.z + c);
                s = __double2float_rn(ag_sv_warp_d(t));
            }
            if (MODE == AG_MODE_DD && __any_sync(0xffffffffu, tag))
                s = __uint_as_float(__float_as_uint(s) | 0x80000000u);
            if (lane == 0)
                finish(at, h.x, s, rp, od);
        }
    }

    /* every unit and hub chunk of a pass, long chains first */
    template <bool LOW> __device__ __forceinline__ bool unit_pass()
    {
        const uint32_t w = (tid >> 5) * gridDim.x + blockIdx.x, nw = gridDim.x * (AG_SOLVE_BLK / 32);
        if (EXACT && iter == 0 && q.nhub) {
            for (uint32_t c = w; c < q.nhub; c += nw)
                chunk<true, LOW>(c);
            if (!predict_scan())
                return false;
        }
        const uint32_t nheads = EXACT ? (q.nhrow + 31u) / 32u : 0u;
        /* items longest first, the next one drawn while one runs */
        const uint32_t nlong = nheads + q.nhub + q.nheavy;
        uint32_t t = w;
        while (t < nlong) {
            uint32_t ticket = 0;
            if (lane == 0)
                ticket = atomicAdd(q.sync + AG_SYNC_BIN, 1u);
            if (t < q.nheavy)
                heavy_unit<LOW>(__ldg(q.heavy + t));
            else if (EXACT && t < q.nheavy + nheads)
                heads<LOW>(t - q.nheavy);
            else
                chunk<false, LOW>(t - q.nheavy - nheads);
            t = __shfl_sync(0xffffffffu, ticket, 0) + nw;
        }
        units<LOW>(t - nlong, nw - nlong);
        if (q.nhub) {
            const uint32_t f = flags;
            if (!grid_sync([&] { return f; }))
                return false;
            hub_rows<LOW>();
        }
        return true;
    }

    /* every row of a pass; LOW: it gathers 16-bit contributions.  Two bodies:
     * with the choice at each gather the 16-bit kernels spilled up to 32 bytes.
     * us per 16-bit pass, FAST / EXACT, chosen at each gather -> here: R-MAT 1 M
     * vertices 73 / 89 -> 61 / 73, 4 M 240 / 312 -> 170 / 219; uniform 4 M
     * 168 / 165 -> 152 / 152 */
    template <bool LOW> __device__ __forceinline__ bool work(float *vals)
    {
        if (UNITS)
            return unit_pass<LOW>();
        if (EXACT && iter == 0 && q.nhub && !predict<LOW>(vals))
            return false;
        const uint32_t nall = q.nhb + q.nbins;
        uint32_t k = blockIdx.x + sub * gridDim.x;
        while (k < nall) {
            /* the next bin's ticket is drawn while this one runs */
            uint32_t ticket = 0;
            if (st == 0)
                ticket = atomicAdd(q.sync + AG_SYNC_BIN, 1u);
            if (k < q.nhb)
                hub_bin<LOW>(k, vals);
            else
                row_bin<LOW>(k - q.nhb, vals);
            if (st == 0)
                sh.next[sub] = ticket + gridDim.x * AG_SUBS;
            ag_sv_sub_sync(sub);
            k = sh.next[sub];
            ag_sv_sub_sync(sub);
        }
        return true;
    }

    /* --------------------------------------------------------------- pass */
    __device__ __forceinline__ bool pass(float *vals)
    {
        start_pass();
        wait_hot();
        if (!(PREC != 0 && low() ? work<true>(vals) : work<false>(vals)))
            return false;
        if (MODE == AG_MODE_SPMV) {
            leave();
            return true;
        }
        /* CTA totals, then the last CTA closes the pass */
        {
            const double e = ag_sv_warp_d(my_err);
            const uint32_t a = __reduce_add_sync(0xffffffffu, my_active);
            my_err = 0.0;
            my_active = 0;
            if (lane == 0) {
                sh.redd[tid >> 5] = e;
                sh.redu[tid >> 5] = a;
            }
            __syncthreads();
            if (tid < 32) {
                const double be = ag_sv_warp_d(sh.redd[tid]);
                const uint32_t ba = __reduce_add_sync(0xffffffffu, sh.redu[tid]);
                if (tid == 0) {
                    if (be != 0.0)
                        atomicAdd(&p.ctl->err_acc, be);
                    if (ba)
                        atomicAdd(&p.ctl->active_acc, ba);
                }
            }
        }
        const bool ok = grid_sync([&] { return MODE == AG_MODE_MULTI ? close_multi() : close_pass(); });
        ++iter;
        return ok;
    }

    /* the pass's record and the stop test, on the last CTA */
    __device__ __forceinline__ uint32_t close_pass()
    {
        if (tid != 0)
            return 0;
        AgControl *c = p.ctl;
        volatile AgControl *vc = c;
        const uint32_t P = iter;
        const uint32_t active = vc->active_acc;
        const double sum = vc->err_acc, err = sum / (double)p.N;
        const uint32_t max_iter = vc->max_iter;
        if (P < AG_MAX_HISTORY) {
            c->hist_active[P] = active;
            c->hist_err[P] = err;
            c->hist_t[P] = ag_globaltimer();
        }
        bool conv = active == 0;
        uint32_t f = 0;
        if (PREC != 0) {
            const bool read_low = (flags & AG_GEN_READ_LOW) != 0, write_low = (flags & AG_GEN_WRITE_LOW) != 0;
            bool next_write = write_low;
            if (read_low)
                c->low_passes = vc->low_passes + 1;
            /* leave 16-bit storage once the residual is small, once it stops
             * falling, or once the 16-bit map has reached its fixed point */
            if (next_write && (err < vc->switch_residual || conv || (P >= 2 && err >= 0.98 * vc->prev_err)))
                next_write = false;
            /* convergence only counts on FP32 contributions */
            if (read_low)
                conv = false;
            c->mode_read = write_low ? 1u : 0u;
            c->mode_write = next_write ? 1u : 0u;
            if (!write_low && vc->switch_pass == 0)
                c->switch_pass = P + 1;
            f |= (write_low ? AG_GEN_READ_LOW : 0u) | (next_write ? AG_GEN_WRITE_LOW : 0u);
        }
        c->prev_err = err;
        c->last_err_sum = sum;
        c->last_err = err;
        c->last_active = active;
        c->iter = P + 1;
        c->converged = conv ? 1u : 0u;
        const bool cont = !conv && (P + 1 < max_iter);
        c->active_acc = 0;
        c->err_acc = 0.0;
        c->stop = cont ? 0u : 1u;
        return f | (cont ? 0u : AG_GEN_STOP);
    }

    /* union of graphs: every thread of the last CTA closes some graphs' pass */
    __device__ __forceinline__ uint32_t close_multi()
    {
        AgControl *c = p.ctl;
        volatile AgControl *vc = c;
        const uint32_t P = iter, max_iter = vc->max_iter;
        int running = 0;
        for (uint32_t g = tid; g < p.ngraphs; g += blockDim.x) {
            if (*((volatile uint32_t *)(p.g_done + g)))
                continue;
            const uint32_t a = *((volatile uint32_t *)(p.g_active + g));
            const uint32_t np = *((volatile uint32_t *)(p.g_passes + g)) + 1;
            const double n_g = (double)(__ldg(p.gstart + g + 1) - __ldg(p.gstart + g));
            p.g_passes[g] = np;
            p.g_err_last[g] = *((volatile double *)(p.g_err + g)) / (n_g > 0 ? n_g : 1.0);
            p.g_active[g] = 0;
            p.g_err[g] = 0.0;
            if (a == 0) {
                p.g_conv[g] = 1;
                p.g_done[g] = 1;
            } else if (np >= max_iter) {
                p.g_done[g] = 1;
            } else {
                running = 1;
            }
        }
        __threadfence();
        running = __syncthreads_or(running);
        if (tid == 0) {
            if (P < AG_MAX_HISTORY)
                c->hist_t[P] = ag_globaltimer();
            c->iter = P + 1;
            c->converged = running ? 0u : 1u;
            c->stop = running ? 0u : 1u;
        }
        return running ? 0u : AG_GEN_STOP;
    }

    /* ------------------------------------------------------ init, normalise */
    /* r = base (or the warm start), first contributions, control reset */
    __device__ __forceinline__ void init(const AgRunConfig &run)
    {
        const uint32_t n = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + tid;
        for (uint64_t v = t0; v < p.N; v += n) {
            /* device row v is caller vertex perm[v]; the warm start is in caller order */
            const float r0 = run.use_init ? p.init_ranks[p.perm ? p.perm[v] : v] : p.base;
            p.rank[UNITS ? q.posof[v] : (uint32_t)v] = r0;
            const uint32_t od = p.outdeg[v];
            const float c = od ? __fdiv_rn(r0, __uint2float_rn(od)) : 0.0f;
            if (PREC != 0)
                ag_st_keep_u16(p.c16_0 + v, ag_sv_to_low<PREC>(c), pol_last);
            else
                ag_st_keep_f32(p.c32_0 + v, c, pol_last);
        }
        for (uint32_t g = t0; g < p.ngraphs; g += n) {
            p.g_active[g] = 0;
            p.g_err[g] = 0.0;
            p.g_done[g] = (run.max_iter > 0 && p.gstart[g + 1] > p.gstart[g]) ? 0u : 1u;
            p.g_passes[g] = 0;
            p.g_conv[g] = 0;
            p.g_err_last[g] = 0.0;
        }
        if (t0 == 0) {
            AgControl *c = p.ctl;
            c->iter = 0;
            c->max_iter = run.max_iter;
            c->active_acc = 0;
            c->done_ctas = 0;
            c->err_acc = 0.0;
            c->eps = run.eps;
            c->converged = 0;
            c->mode_read = PREC != 0 ? 1u : 0u;
            c->mode_write = PREC != 0 ? 1u : 0u;
            c->switch_pass = 0;
            c->switch_residual = run.switch_residual;
            c->prev_err = 1e300;
            c->rank_sum = 0.0;
            c->use_init = run.use_init;
            c->low_passes = 0;
            c->t0 = ag_globaltimer();
            c->stop = (run.max_iter > 0 && p.N > 0) ? 0u : 1u;
            c->fault = 0;
        }
    }

    /* ranks / N in binary32 (pageRank.c:1079-1085), back in caller order, FP64 sum */
    __device__ __forceinline__ void normalise()
    {
        const float fN = __uint2float_rn(p.N);
        double sum = 0.0;
        for (uint64_t v = blockIdx.x * blockDim.x + tid; v < p.N; v += gridDim.x * blockDim.x) {
            float div = fN;
            if (MODE == AG_MODE_MULTI) {
                /* each graph of a union is normalised by its own vertex count */
                const uint32_t g = graph_of((uint32_t)v);
                div = __uint2float_rn(__ldg(p.gstart + g + 1) - __ldg(p.gstart + g));
            }
            /* caller vertex v, or the vertex of position v */
            uint32_t at = (uint32_t)v, to = (uint32_t)v;
            if (UNITS) {
                to = (at & ~(AG_UNIT_WIN - 1u)) + AG_UNIT_ROW(q.info[at]);
                to = p.perm ? p.perm[to] : to;
            } else if (p.inv) {
                at = p.inv[v];
            }
            const float r = __fdiv_rn(ag_ld_rank(p.rank + at), div);
            p.out[to] = r;
            sum += (double)r;
        }
        sum = ag_sv_warp_d(sum);
        if (lane == 0)
            sh.redd[tid >> 5] = sum;
        __syncthreads();
        if (tid < 32) {
            sum = ag_sv_warp_d(sh.redd[tid]);
            if (tid == 0)
                atomicAdd(&p.ctl->rank_sum, sum);
        }
    }
};

template <int MODE, int PREC, bool EXACT, bool UNITS>
__global__ void __launch_bounds__(AG_SOLVE_BLK, 1) ag_solve_kernel(const AgSolveParams q, const AgRunConfig run)
{
    __shared__ AgSvShared sh;
    AgSolve<MODE, PREC, EXACT, UNITS> s(q, sh);
    float *vals = reinterpret_cast<float *>(ag_sv_dyn + (size_t)q.p.hot_n * 4) + (size_t)s.sub * q.buf;
    if (threadIdx.x == 0)
        ag_sv_mbar_init(&sh.mbar);
    /* a graph that was given up stays so until the host has cleared its words:
     * the barrier that a solve begins with does not open then; other launches
     * ask here (all threads together, the mark may be set just now) */
    s.gen = *((volatile uint32_t *)(q.sync + AG_SYNC_GEN));
    bool ok = true;
    if (MODE == AG_MODE_SPMV) {
        s.iter = 0;
        s.eps = 0.0;
        s.flags = 0;
        if (q.x_in) {
            const uint32_t n4 = q.p.N / 4u, t0 = blockIdx.x * blockDim.x + threadIdx.x;
            for (uint32_t v = t0; v < n4; v += gridDim.x * blockDim.x) {
                const uint4 i = __ldg(reinterpret_cast<const uint4 *>(q.p.perm) + v);
                const float4 x = make_float4(__ldg(q.x_in + i.x), __ldg(q.x_in + i.y), __ldg(q.x_in + i.z),
                                             __ldg(q.x_in + i.w));
                reinterpret_cast<float4 *>(q.x_dev)[v] = x;
            }
            if (t0 < (q.p.N & 3u))
                q.x_dev[4u * n4 + t0] = __ldg(q.x_in + __ldg(q.p.perm + 4u * n4 + t0));
            s.gen &= ~AG_GEN_ABORT;
            ok = s.grid_sync([&] { return 0u; });
        } else {
            ok = !__syncthreads_or(s.gen & AG_GEN_ABORT);
        }
        ok = ok && s.pass(vals);
    } else {
        if (q.do_init) {
            s.gen &= ~AG_GEN_ABORT;
            s.init(run);
            const uint32_t f = (run.max_iter > 0 && q.p.N > 0 ? 0u : AG_GEN_STOP) |
                               (PREC != 0 ? AG_GEN_READ_LOW | AG_GEN_WRITE_LOW : 0u);
            s.iter = 0;
            s.eps = run.eps;
            ok = s.grid_sync([&] { return f; });
        } else {
            ok = !__syncthreads_or(s.gen & AG_GEN_ABORT);
            volatile AgControl *c = q.p.ctl;
            s.iter = c->iter;
            s.eps = c->eps;
            s.flags = (c->stop ? AG_GEN_STOP : 0u) | (c->mode_read ? AG_GEN_READ_LOW : 0u) |
                      (c->mode_write ? AG_GEN_WRITE_LOW : 0u);
        }
        for (uint32_t n = 0; ok && n < q.max_pass && !(s.flags & AG_GEN_STOP); ++n)
            ok = s.pass(vals);
        if (ok && q.do_norm)
            s.normalise();
    }
    if (!ok && threadIdx.x == 0)
        ag_sv_give_up(q.sync, s.gen & ~AG_GEN_ABORT, gridDim.x, q.gave_up);
}

template <int MODE, int PREC, bool UNITS> static const void *solve_ptr(int exact)
{
    return exact ? (const void *)ag_solve_kernel<MODE, PREC, true, UNITS>
                 : (const void *)ag_solve_kernel<MODE, PREC, false, UNITS>;
}

extern "C" const void *ag_solve_kernel_ptr(int mode, int prec, int exact, int units)
{
    if (mode == AG_MODE_MULTI)
        return solve_ptr<AG_MODE_MULTI, 0, false>(exact);
    if (mode == AG_MODE_SPMV)
        return units ? solve_ptr<AG_MODE_SPMV, 0, true>(exact) : solve_ptr<AG_MODE_SPMV, 0, false>(exact);
    if (mode == AG_MODE_DD)
        return units ? solve_ptr<AG_MODE_DD, 0, true>(exact) : solve_ptr<AG_MODE_DD, 0, false>(exact);
    if (units)
        return prec == 1   ? solve_ptr<AG_MODE_PR, 1, true>(exact)
               : prec == 2 ? solve_ptr<AG_MODE_PR, 2, true>(exact)
                           : solve_ptr<AG_MODE_PR, 0, true>(exact);
    return prec == 1   ? solve_ptr<AG_MODE_PR, 1, false>(exact)
           : prec == 2 ? solve_ptr<AG_MODE_PR, 2, false>(exact)
                       : solve_ptr<AG_MODE_PR, 0, false>(exact);
}
