/*
 * ag_solve.h -- parameters of the solve kernel (ag_solve.cu).
 */
#ifndef AG_SOLVE_H
#define AG_SOLVE_H

#include "ag_units.h"
#include "ag_device.h"

#ifndef AG_SUBS
#define AG_SUBS 2             /* warp groups of a CTA, each on its own bin      */
#endif
#define AG_SOLVE_BLK 1024
#define AG_SUB_THREADS (AG_SOLVE_BLK / AG_SUBS)
#define AG_SUB_WARPS (AG_SUB_THREADS / 32)

/* words of AgSolveParams::sync */
#define AG_SYNC_COUNT 0       /* CTAs that have arrived at a barrier, how many
                                 barriers were opened << 12, AG_COUNT_ABORT     */
#define AG_SYNC_GEN 1         /* barriers passed << 4 | flags                   */
#define AG_SYNC_BIN 2         /* bins handed out in this pass                   */
#define AG_SYNC_KEPT 3        /* rounds kept in this pass                       */
#define AG_SYNC_WORDS 4
#define AG_KEPT_QUADS 96u     /* 16-byte words of a kept round                  */
#define AG_GEN_STOP 1u
#define AG_GEN_READ_LOW 2u
#define AG_GEN_WRITE_LOW 4u
#define AG_GEN_ABORT 8u       /* a CTA gave up waiting: no barrier of the graph
                                 opens again until the host has cleared the
                                 words                                          */
#define AG_COUNT_ABORT 0x80000000u
#define AG_COUNT_CTAS 0xfffu
#define AG_GEN_SHIFT 4

typedef struct AgSolveParams
{
    AgPullParams p;
    const AgBin *bins;
    const uint4 *hubs;
    const uint32_t *brow, *ubase, *ids;
    const float *w;           /* weights in the order of ids (SpMV)             */
    const float *x_in;        /* SpMV: the vector in caller order, to be put in
                                 device order in x_dev first (NULL: p.x is)     */
    float *x_dev, *y;         /* SpMV: y in caller order                        */
    uint32_t nbins, nhub;     /* row bins, hub chunks                           */
    uint32_t per_bin, nhb;    /* hub chunks per bin, bins they make             */
    uint32_t buf;             /* floats of a group's buffer                     */
    /* units (nunits 0: bins): ids, hubs, nhub and the hub_* arrays are theirs */
    uint32_t nunits, nhrow, nheavy, heavy_quads, nbatch;
    const uint32_t *heavy, *bstart;
    const uint32_t *info, *uoutdeg, *posof, *hrow;
    const uint32_t *ubaseq;   /* AgUnitPlan::ubase                              */
    const uint4 *uids;        /* the units' quads                               */
    double *hub_sum;          /* per chunk: FAST partial sum, EXACT head sum    */
    uint4 *hub_words;         /* EXACT: per round its two maps and where its
                                 values are kept                                */
    uint16_t *hub_pred;       /* EXACT: the sum at each round's start, top half */
    float4 *kept;             /* EXACT: lanes' maps (512 bytes) and values (1 KB)
                                 of the rounds that should leave a binade       */
    uint32_t kept_cap;        /* rounds it can hold                             */
    uint32_t *hub_seen;       /* bins, per chunk (at a row's first): chunks done      */
    uint32_t *hub_tag;        /* units, data-driven: a sign was set; 2 x nhub    */
    uint32_t *sync;           /* AG_SYNC_WORDS                                  */
    uint32_t spins;           /* polls of a grid barrier before it gives up     */
    volatile uint32_t *gave_up; /* page-locked word that the CTA which gives up
                                 sets to 1                                      */
    uint32_t do_init, do_norm, max_pass; /* parts of a solve in this launch     */
} AgSolveParams;

#ifdef __cplusplus
extern "C" {
#endif
const void *ag_solve_kernel_ptr(int mode, int prec, int exact, int units);
#ifdef __cplusplus
}
#endif

#endif /* AG_SOLVE_H */
