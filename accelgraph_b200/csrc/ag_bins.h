/*
 * ag_bins.h -- the solve kernel's work layout ("bins"), planned on the device
 * once per graph by ag_bins.cu and run by ag_solve.cu.
 *
 * A bin is one group of warps' unit of work: a window of consecutive rows
 * whose in-edges (those of rows above AG_BIN_HUB in-edges aside) fit its
 * shared-memory buffer.  The bin's in-neighbour ids are copied into the order
 * in which the kernel stages them ("slots"):
 *   long rows  (AG_BIN_SEQ < degree <= AG_BIN_HUB), longest first: each row's
 *              ids in stream order, padded to a multiple of 4 slots;
 *   short rows (1 .. AG_BIN_SEQ in-edges), longest first, 32 to a unit: slot
 *              32 i + l of a unit is the i-th id of its row l, so that a warp
 *              that sums one row per lane reads 32 neighbouring words;
 * padding slots hold id 0 and are never summed.  `brow` lists the rows in that
 * order (local row | degree << 16, 32 entries to a unit, empty entries 0) and
 * `ubase` each unit's first slot.
 * Rows above AG_BIN_HUB in-edges are cut into chunks of AG_BIN_HUB slots, in
 * stream order, the last one padded.
 */
#ifndef AG_BINS_H
#define AG_BINS_H

#include <cuda_runtime.h>
#include <stdint.h>

#include "ag_device.h"

#define AG_BIN_SEQ 32u     /* short rows: summed in stream order in either order */
#define AG_BIN_HUB 2048u   /* in-edges of a hub chunk; longer rows are hub rows  */
#define AG_BIN_ROUND 256u  /* values of an EXACT-order hub round                 */
#define AG_BIN_ROUNDS (AG_BIN_HUB / AG_BIN_ROUND)
#define AG_BIN_HEAD 512u   /* EXACT order: a hub row's first values, one lane    */
#define AG_BIN_PAD (32u * AG_BIN_SEQ) /* most padding slots of a bin's short rows */
/* a bin's rows weigh less than quantum + (AG_BIN_HUB + 4) together, a row's
 * weight being its slots (long rows with their padding) + 1; the buffer holds
 * the slots and one sum per row, and 16 floats that a lane's chain may load
 * past its row */
#define AG_BIN_BUF(q) (((q) + AG_BIN_HUB + 4u + AG_BIN_PAD + 16u + 63u) & ~63u)

/* one bin (two uint4) */
typedef struct AgBin
{
    uint32_t r0, nrows;    /* window of device rows                          */
    uint32_t nlong, nshort;
    uint32_t nslots, gid;  /* slots; graph of a union                        */
    uint64_t sbase;        /* first slot                                     */
} AgBin;

/* one hub chunk (uint4): row, chunk index in the row, the row's first chunk,
 * chunk in-edges - 1 | the row's chunks << 11 */

typedef struct AgBinPlan
{
    uint32_t quantum, buf;     /* row weight per bin; buffer floats            */
    uint32_t nbins, nhub;      /* row bins; hub chunks                         */
    uint64_t nslots;
    AgBin *bins;
    uint4 *hubs;
    uint32_t *brow, *ubase;
    uint32_t *ids;             /* in slot order, hub chunks first              */
    float *w;                  /* weights in the same order, or NULL           */
    uint64_t *pre;             /* planning: scanned weights (and hub chunks)   */
    void *tmp;
} AgBinPlan;

#ifdef __cplusplus
extern "C" {
#endif
/* weights of the rows and their scan; *total_host receives the totals (hub
 * chunks << 40 | weight) once the stream has been waited for */
cudaError_t ag_bins_count(const uint32_t *row_off, uint32_t n, AgBinPlan *b, uint64_t *total_host, cudaStream_t s);
/* sizes from the totals: nbins, nhub, nslots, buf */
void ag_bins_shape(AgBinPlan *b, uint64_t total, uint32_t quantum, uint32_t ngraphs);
/* bins, rows and hub chunks (the caller has allocated bins, hubs, brow, ubase) */
cudaError_t ag_bins_rows(const uint32_t *row_off, uint32_t n, const uint32_t *gstart, uint32_t ngraphs, AgBinPlan *b,
                         cudaStream_t s);
/* in-neighbour ids (and weights) in slot order */
cudaError_t ag_bins_ids(const uint32_t *row_off, const uint32_t *ids, const float *w, const AgBinPlan *b,
                        cudaStream_t s);
size_t ag_bins_brow_words(const AgBinPlan *b, uint32_t n);
#ifdef __cplusplus
}
#endif

/* first entry of bin k's rows in brow (a multiple of 32) */
__host__ __device__ __forceinline__ uint32_t ag_bin_list(uint32_t r0, uint32_t k)
{
    return (r0 & ~31u) + 96u * k;
}

#endif /* AG_BINS_H */
