/*
 * ag_units.h -- the solve kernel's layout of a large graph ("units"), planned
 * on the device once per graph by ag_units.cu and run by ag_solve.cu.
 *
 * Rows are sorted by their quads, longest first, inside windows of AG_UNIT_WIN
 * consecutive device rows; a row's place is its position.  32 consecutive
 * positions are a unit, one warp's work, one row per lane.  A unit's ids are
 * stored in quads: quad 32 i + l holds ids 4 i .. 4 i + 3 of its row l, so a
 * warp reads 512 neighbouring bytes and every lane gets four ids of its own
 * row.  A unit has as many quads per row as its longest row needs; padding ids
 * are 0.  Ranks and out-degrees are kept by position, contributions by device
 * row (their order decides the hot table).
 * Rows above `longest` in-edges (hub rows) take a position but no quads:
 * their ids are copied in stream order to chunks of AG_BIN_HUB slots, the
 * last one padded.
 */
#ifndef AG_UNITS_H
#define AG_UNITS_H

#include "ag_bins.h"

#define AG_UNIT_WIN 2048u
#define AG_UNIT_COST 2u     /* a unit's fixed work, in quads per row            */
#define AG_UNIT_LONG 2047u  /* longest row a unit can hold                      */
/* info of a position: local row in the window | in-degree << 11, or for a
 * hub row the top bit */
#define AG_UNIT_ROW(x) ((x) & (AG_UNIT_WIN - 1u))
#define AG_UNIT_LEN(x) (((x) >> 11) & 0xfffu)
#define AG_UNIT_HUB 0x80000000u

typedef struct AgUnitPlan
{
    uint32_t nunits, longest;
    uint32_t heavy_quads;  /* units of more quads per row are run first       */
    uint32_t batch;        /* weight of a batch of the other units; a unit
                              weighs its quads per row + AG_UNIT_COST         */
    uint32_t nbatch;
    uint32_t *bstart;      /* first unit of each batch, + end                 */
    uint32_t nhub, nhrow;  /* hub chunks, hub rows                            */
    uint64_t quads;        /* of the units                                    */
    uint32_t *info;        /* per position                                    */
    uint32_t *ubase;       /* per unit: its first quad, + end                 */
    uint32_t *heavy;       /* units of more than heavy_quads quads per row     */
    uint32_t nheavy;
    uint32_t *outdeg;      /* per position                                    */
    uint32_t *posof;       /* position of a device row                        */
    uint4 *hubs;           /* hub chunks, as in ag_bins.h                     */
    uint32_t *hrow;        /* first chunk of each hub row                     */
    uint4 *ids;            /* hub chunks, then the units' quads               */
    float4 *w;             /* weights in the same order, or NULL              */
    uint32_t *cnt;         /* planning: hub chunks, hub rows, heavy units     */
    void *tmp;
} AgUnitPlan;

#ifdef __cplusplus
extern "C" {
#endif
/* positions and unit sizes (the caller has set longest and allocated info,
 * ubase, heavy, outdeg, posof, cnt); totals_host receives hub chunks, hub
 * rows, heavy units and quads once the stream has been waited for */
cudaError_t ag_units_rows(const uint32_t *row_off, const uint32_t *outdeg, uint32_t n, AgUnitPlan *u,
                          uint32_t *totals_host, cudaStream_t s);
/* batches of units that hold `quads` quads: their number */
uint32_t ag_units_batches(const AgUnitPlan *u, uint64_t quads);
/* hub chunks, batches and ids (the caller has allocated hubs, hrow, bstart,
 * ids and set nbatch) */
cudaError_t ag_units_ids(const uint32_t *row_off, const uint32_t *ids, const float *w, uint32_t n, const AgUnitPlan *u,
                         cudaStream_t s);
#ifdef __cplusplus
}
#endif

#endif /* AG_UNITS_H */
