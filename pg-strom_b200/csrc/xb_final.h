/*
 * xb_final.h
 *
 * The final-stage kernels of the device translation unit (xb_exec.cu) and
 * their arguments: kds_final materialisation, GPU-Sort of the groups, the
 * merge of another kds_final into a session's group table and the
 * inner-buffer rebuild.  The host services that launch them live in
 * xb_final.cu (xpuB200Final, xpuB200FinalNoAlloc, xpuB200MergeFinal,
 * xpuB200FinalParts, xpuB200InnerRebuild).  Internal; the public interface
 * is include/xpu_b200.h.
 */
#ifndef XB_FINAL_H
#define XB_FINAL_H

#include <cuda_runtime.h>
#include <cstdint>
#include "xb_plan.h"
#include "xb_exec_dev.cuh"
#include "xb_sort.cuh"

#define XB_GENT_MAX     2048    /* largest group entry a merge stages per thread */

/* the tuple of a group whose size and attribute offsets are the plan's
 * alone (every key fixed-width of 4 or 8 bytes, none NULL), as 4-byte
 * units: what each one is made of */
enum {
    XB_FU_CONST = 0,                /* imm */
    XB_FU_COPY,                     /* 4 bytes of the entry */
    XB_FU_ROWID,
    XB_FU_SUM_LO, XB_FU_SUM_HI,     /* float8 sum + its compensation */
    XB_FU_MM_ATTRS,                 /* min/max: valid flag */
    XB_FU_MMFP_LO, XB_FU_MMFP_HI,   /* float8 min (imm 0) / max (imm 1) */
    XB_FU_NUM_ATTRS,                /* numeric: imm | special flags */
    XB_FU_FLT4,                     /* float8 image of a float4 key */
};
#define XB_FINAL_UNITS  128
struct XbFinalProg {
    uint32_t        nunits;         /* even; 0: the plan has no fixed tuple */
    uint32_t        item;           /* bytes of an item, hash link included */
    struct { uint16_t op, src; uint32_t imm; } unit[XB_FINAL_UNITS];
};

/* one hash partition of the groups, being written as a kds_final */
struct XbFinalPart {
    uint64_t        out;            /* its start in the output buffer */
    uint64_t        items_base;     /* offset of the first item in the part */
    uint64_t        length;
    uint32_t        nslots;
    uint32_t        nitems;
};

/* kds_final by tiles of the group table: the groups and item bytes of
 * every (part, tile), then the tuples (xb_final_tiles, xb_final_fill) */
#define XB_FINAL_TILE   256
#define XB_FINAL_SMALL  16384       /* slots of a table that one CTA counts */
#define XB_FINAL_PARTS  1024        /* parts of one launch (their counters are in shared memory) */
struct XbTileArgs {
    const xb_plan  *plan;
    const xb_gtable *gt;
    uint64_t        cap;
    uint32_t        tile_slots;     /* a multiple of XB_FINAL_TILE */
    uint32_t        ntiles;
    uint32_t        nparts;         /* of all: part = hash % nparts */
    uint32_t        part0;          /* the parts [part0, part0 + pset) are this launch's */
    uint32_t        pset;
    uint32_t        row_format;
    uint32_t       *count;          /* [(part - part0) * ntiles + tile] */
    uint64_t       *bytes;
    const uint32_t *count_scan;     /* exclusive prefixes of the two, over all parts */
    const uint64_t *bytes_scan;
    char           *out;
    const XbFinalPart *part;        /* nullptr: the one part 'only' */
    XbFinalPart     only;
    const uint64_t *head;           /* the session's kds_final definition */
    uint32_t        head_len;
    const uint32_t *list;           /* the entries to write, in order (cap of them), or
                                     * nullptr: every group, in table order */
    XbFinalProg     prog;
};

/* GPU-Sort: the sort keys of the ready groups, as radix words */
struct XbSortArgs {
    const xb_plan  *plan;
    const xb_gtable *gt;
    const uint32_t *ents;           /* per rank: entry index */
    uint64_t       *keyw;           /* word w of key k at keyw[(2k + w) * n + r] */
    uint8_t        *nul;            /* NULL flag of key k at nul[k * n + r] */
    uint32_t        n;
};

/* the first 'want' groups by their first sort key: radix selection of its
 * leading XB_TOP_BITS bits (the NULL flag, then the key's high word) by
 * digits of 11 bits, then every group up to and including the last one's
 * digits */
#define XB_TOP_DIGITS   4
#define XB_TOP_BINS     2048
#define XB_SORT_SMALL   4096        /* groups that one CTA sorts */
struct XbTopArgs {
    const uint64_t *hi;             /* first key's high words and NULL flags */
    const uint8_t  *nul;
    uint32_t        n;
    uint32_t       *hist;           /* XB_TOP_DIGITS * XB_TOP_BINS, zero */
    uint64_t       *prefix;         /* [0] digits chosen so far, [1] groups still wanted */
    uint32_t       *cand;           /* the groups picked, XB_SORT_SMALL at most */
    uint32_t       *ncand;          /* how many there are */
};

/* groups kept, in order: LIMIT, or the window rank of each group within
 * its partition (row_number / rank / dense_rank) against its limit */
struct XbRankArgs {
    const xb_plan  *plan;
    const uint32_t *idx;            /* rank of the group at each sorted position */
    const uint64_t *keyw;
    const uint8_t  *nul;
    uint32_t        n;
    uint32_t       *part_start;     /* position that starts a new partition, else 0 */
    uint32_t       *peer_start;     /* position that starts a new peer group, else 0 */
    uint32_t       *peer_flag;      /* 1 where a peer group starts */
};

struct XbKeepArgs {
    const xb_plan  *plan;
    const uint32_t *idx;
    const uint32_t *ents;
    uint32_t        n;
    const uint32_t *part_start;     /* after the max-scan: the partition's first position */
    const uint32_t *peer_start;     /* after the max-scan */
    const uint32_t *peer_cnt;       /* inclusive sum of peer_flag */
    uint32_t       *keep_flag;
};

/* merge of another kds_final into the session's group table */
struct XbMergeArgs {
    const xb_plan          *plan;
    const kern_data_store  *kds;        /* the other kds_final (device copy) */
    xb_gtable              *gt;
    xb_status              *st;
};

/* inner-buffer rebuild into a KDS_FORMAT_HASH buffer */
struct XbRebuildArgs {
    kern_data_store        *dst;
    const kern_data_store  *src;
    uint64_t                dst_head;   /* KDS_HEAD_LENGTH(dst) */
    uint64_t                src_rowidx; /* offset of src's row index */
    uint32_t                divisor;    /* 0: every row */
    uint32_t                remainder;
    uint32_t               *overflow;
};

/* the kernels (xb_exec.cu) */
__global__ void __launch_bounds__(XB_FINAL_TILE) xb_final_tiles(const __grid_constant__ XbTileArgs a);
__global__ void __launch_bounds__(XB_FINAL_TILE) xb_final_scan_small(XbTileArgs a, uint32_t *count_scan,
                                                                      uint64_t *bytes_scan, uint32_t n);
__global__ void __launch_bounds__(1024) xb_final_count_small(const __grid_constant__ XbTileArgs a, uint64_t *totals);
__global__ void xb_final_totals(XbTileArgs a, uint64_t *totals);
__global__ void xb_final_heads(const __grid_constant__ XbTileArgs a);
__global__ void __launch_bounds__(XB_FINAL_TILE) xb_final_fill(const __grid_constant__ XbTileArgs a);
__global__ void __launch_bounds__(XB_FINAL_TILE) xb_final_ents(const __grid_constant__ XbTileArgs a, uint32_t *ents);
__global__ void xb_top_hist(XbTopArgs a, uint32_t digit);
__global__ void __launch_bounds__(XB_SCAN_BLOCK) xb_top_select(XbTopArgs a, uint32_t digit);
__global__ void xb_top_gather(XbTopArgs a);
__global__ void __launch_bounds__(1024) xb_sort_small(XbSortArgs a, const uint32_t *cand, uint32_t m, uint32_t *idx);
__global__ void xb_sort_keys(XbSortArgs a);
__global__ void xb_sort_pass_key64(const uint64_t *col, const uint32_t *idx, uint64_t *out, uint32_t n);
__global__ void xb_sort_pass_key8(const uint8_t *col, const uint32_t *idx, uint8_t *out, uint32_t n);
__global__ void xb_sort_bounds(XbRankArgs a);
__global__ void xb_sort_keepflag(XbKeepArgs a);
__global__ void xb_sort_keep(XbKeepArgs a, const uint32_t *keep_scan, uint32_t *list);
__global__ void xb_iota_u32(uint32_t *out, uint32_t n);
__global__ void __launch_bounds__(XB_BLOCK) xb_merge_final(XbMergeArgs args);
__global__ void __launch_bounds__(XB_BLOCK) xb_inner_rebuild(XbRebuildArgs args);

/* 256-byte alignment of the work arrays carved from one buffer */
static inline uint64_t xb_align256(uint64_t x)
{
    return (x + 255) & ~255ULL;
}

#endif  /* XB_FINAL_H */
