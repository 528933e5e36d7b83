/*
 * Host-side index algebra of the compact sparse-grid layout and the device
 * layout derived from it.  Plain C, shared by the API (sgrid.c) and the CUDA
 * launchers.
 *
 * Device layout ("group-aligned compact layout"): exactly the reference's
 * compact order (adaptive_sparse_grid_bench.c:130-140, 187-207), except that
 * each level group starts on a 32-element boundary.  A subspace of group
 * s >= 2 therefore starts on a 16-byte boundary (FP32), which is what the
 * bulk-copy engine and vector loads need.  Compact index j of group s maps to
 * device index j - lidx[s] + plidx[s].
 */
#ifndef SG_LAYOUT_H
#define SG_LAYOUT_H

#include <stdint.h>

#include "../../include/sgrid.h"

#ifdef __cplusplus
extern "C" {
#endif

#define SG_GROUP_ALIGN 32 /* elements */

typedef struct sg_layout {
    int d, n;
    int lim[SG_MAX_DIMS];
    int64_t dp[SG_MAX_DIMS][SG_MAX_LEVELS]; /* dp[i][s], c:113-129          */
    int64_t lidx[SG_MAX_LEVELS + 1];        /* compact group offsets        */
    int64_t plidx[SG_MAX_LEVELS + 1];       /* device (padded) group offsets */
    int64_t N, S, Npad;
    int64_t Nblk;  /* slots of the evaluation (block) layout             */
    int64_t nrows; /* rows of dim B in it (level vectors of dims 0..d-2) */
} sg_layout;

/* One 1-D "chain" of sweep k: the subspaces that differ only in l_k.  They
 * hold 2^sigma independent poles (one per index combination of the other
 * dims); segment j (l_k = j) is the whole subspace, 2^(sigma+j) values. */
typedef struct sg_chain {
    uint32_t seg;   /* first entry of this chain in the segment-offset array */
    uint8_t sigma;  /* sum of the other dims' levels                         */
    uint8_t lmax;   /* highest l_k in the chain (>= 1; lmax 0 needs no work) */
    uint8_t lo;     /* sum of the levels of dims k+1..d-1 (index bits below) */
    uint8_t pad;
} sg_chain;

int sg_layout_init(sg_layout *L, int d, int n, const int *limits);
int64_t sg_layout_l2idx(const sg_layout *L, const int *lv);
void sg_layout_idx2l(const sg_layout *L, int64_t pos, int s, int *lv);
int64_t sg_layout_gp2idx(const sg_layout *L, const int *lv, const int *ix);
int sg_layout_idx2gp(const sg_layout *L, int64_t idx, int *lv, int *ix);
/* Device offset of the subspace with level vector lv. */
int64_t sg_layout_subspace_offset(const sg_layout *L, const int *lv);

/* Chains of sweep k with lmax >= 1, largest first.  *chains and *seg_off are
 * malloc'd; seg_off[c.seg + j] is the device offset of segment j. */
int sg_layout_chains(const sg_layout *L, int k, sg_chain **chains, int64_t *nchains,
                     uint32_t **seg_off, int64_t *nseg);


/* ---- passes of several sweeps (hier_fused.cu) ---------------------------
 * A pass runs the sweeps of dims k0..k0+g-1.  A unit holds the subspaces that
 * differ only in those dims' levels: 2^sigma cells of a g-dimensional grid of
 * budget R.  The nodes of that grid are numbered by level sum, so the grid of
 * a smaller budget is a prefix. */
typedef struct sg_unit {
    uint32_t off;  /* first of its subspace offsets, one per combo of sum <= R */
    uint8_t R;     /* level budget of the pass's dims                          */
    uint8_t sigma; /* level sum of the other dims                              */
    uint8_t lo;    /* of those after the pass's dims                           */
    uint8_t pad;
} sg_unit;
typedef struct sg_unit_combo { /* levels of the pass's dims */
    uint32_t node;             /* first node                */
    uint8_t lv[3], sum;
} sg_unit_combo;
typedef struct sg_unit_node { /* a point that a sweep updates, and its parents */
    uint16_t node, left, right, pad;
} sg_unit_node;
#define SG_UNIT_NONE 0xFFFF
typedef struct sg_unit_tables {
    const sg_unit_combo *combos; /* device */
    const sg_unit_node *nodes;   /* device: per dim q and level j, ordered by level sum */
    int lmax[3];
    const uint16_t *combo_of;    /* device: the combo of each node */
    int ncombo[SG_MAX_LEVELS], nnode[SG_MAX_LEVELS]; /* combos, nodes of sum <= R  */
    uint32_t first[3][SG_MAX_LEVELS];               /* first entry of (q, j)       */
    uint16_t count[3][SG_MAX_LEVELS][SG_MAX_LEVELS]; /* entries of (q, j) of sum <= R */
} sg_unit_tables;
/* Shared-memory row of a node: its cells, padded against bank conflicts
 * between the nodes that one 16-byte load scatters to. */
#ifdef __CUDACC__
__host__ __device__
#endif
static inline int sgk_unit_stride(int sigma)
{
    return (1 << sigma) + (sigma >= 3 ? 4 : 0);
}
#define SG_UNIT_MAX_BYTES (100 * 1024) /* two CTAs per SM at least */
#define SG_PASS_NODES 10240
#define SG_PASS3_NODES 1100
#define SG_PASS1_BYTES (48 * 1024)
/* The dims a pass from k0 on should run (0: none; the single-dim sweeps do
 * better), for elements of elem_bytes. */
int sg_layout_pass_dims(const sg_layout *L, int k0, int elem_bytes);
/* The pass's tables, all malloc'd (NULL on failure); tables' pointers unset.
 * max_elems: shared-memory elements of its largest unit. */
typedef struct sg_pass_host {
    sg_unit *units;
    uint32_t *offs;
    sg_unit_combo *combos;
    sg_unit_node *nodes;
    uint16_t *combo_of;
    int64_t nunits, noffs, ncombos, nnodes, nall, max_elems;
    sg_unit_tables tables;
} sg_pass_host;
int sg_layout_pass(const sg_layout *L, int k0, int g, sg_pass_host *p);
void sg_layout_pass_free(sg_pass_host *p);
/* Upper bound of the device bytes of all sweep tables. */
int64_t sg_layout_sweep_bytes(const sg_layout *L);

/*
 * Evaluation layout ("block layout").  The same surpluses, ordered for the
 * evaluation walk.  Dims 0..d-4 form the prefix; the three innermost dims are
 * C = d-3, A = d-2, B = d-1 (for d < 3 the missing leading ones are treated
 * as dims with limit 0).  For every prefix level vector p (depth-first
 * order, level ascending) and every cell I of p (row-major over the prefix
 * dims) one block holds all subspaces (p, c, a, b) below the level budget
 * R = n-1-|p|:
 *   planes c = 0..cmax, each 2^c sub-blocks (one per cell t_c of dim C);
 *   a sub-block of budget r = R-c has rows a = 0..amax(r), each 2^a poles
 *   (one per cell t_a of dim A);
 *   a pole holds what a query point needs of dim B's levels b = 0..L (L =
 *   rowlen-1), in one slot or one 8-byte pair per point:
 *     L = 0: the one surplus;
 *     L = 1: per cell t of level 1 the pair (surplus of level 0, surplus of
 *       level 1 in cell t);
 *     L >= 2: the levels summed.  The sum over b of surplus * hat is linear
 *       in x_B on each of the 2^(L+1) halves of the cells of level L; half h
 *       holds the pair (value at its left end, value at its right end minus
 *       that), both summed in FP64 from the surpluses and rounded once.
 * A query point finds the pair of row (c, a) at
 *   base + coff(c) + t_c * sub(R-c) + aoff(R-c, a) + t_a * plen + 2 t_B
 * with t_B its cell of level 1 (L = 1) or its half (L >= 2).  Every row with
 * L >= 1 starts at an even offset (all sizes before it in a block are even),
 * so a pair moves with one 8-byte load.
 */
/* Slots of a pole whose last level of dim B is L. */
#define SG_POLE_SLOTS(L) ((L) == 0 ? 1u : ((L) == 1 ? 4u : 4u << (L)))

typedef struct sg_eval_sub {
    int amax;                         /* last row: min(r, lim_A)           */
    int rowlen[SG_MAX_LEVELS];        /* levels of dim B in row a           */
    uint32_t aoff[SG_MAX_LEVELS + 1]; /* row starts; aoff[amax+1] = size    */
} sg_eval_sub;

typedef struct sg_eval_shape {
    int R, cmax;                      /* budget, last plane min(R, lim_C)   */
    uint32_t coff[SG_MAX_LEVELS + 1]; /* plane starts; coff[cmax+1] = size  */
} sg_eval_shape;

void sg_layout_eval_sub(const sg_layout *L, int r, sg_eval_sub *sh);
void sg_layout_eval_shape(const sg_layout *L, int R, sg_eval_shape *sh);

/* Segments of a point's sum.  The evaluation adds up a point's sum in
 * segments of consecutive blocks of the walk, each with its own compensated
 * sum, the segments of a part (SG_SEG_PER_PART of them) into the part's and the
 * parts into the total.  The bounds depend on the grid alone, so one thread
 * adding everything and many warps adding a few segments each give the same
 * bits.  nseg = 1 for small grids and d < 4; parts = 1 or nseg / SG_SEG_PER_PART.
 * A warp's chain of dependent work is then S / nseg subspaces at the shortest:
 * about 128 of them, below which a segment's walk down from the root costs as
 * much as its sums. */
#define SG_SEG_PER_PART 16
#define SG_SEG_SUBSPACES 128
#define SG_MAX_SEGS (SG_SEG_PER_PART * 8)
#define SG_SEG_UNIT_BUDGET 3 /* the kernels' SG_EVAL_MAX_LEAF2 */
int sg_layout_parts(const sg_layout *L);
int sg_layout_segs(const sg_layout *L);
/* Words of the segment table: the extents in the block layout of the subtree
 * of the walk entered at depth K = 0..d-3 with budget b = 0..n-1, at K*n + b
 * (the walk visits prefix dims 0..d-4, blocks sit at depth d-3), then the
 * nseg+1 bounds as block-layout offsets.  0 when nseg = 1. */
int64_t sg_layout_seg_words(const sg_layout *L);
int sg_layout_seg_table(const sg_layout *L, const uint32_t *blk3, uint32_t *table);

/* Per-row repack descriptor (compact layout -> block layout): the row of
 * one level vector of dims 0..d-2, whose levels 0..L of dim B are L+1
 * subspaces. */
typedef struct sg_repack {
    uint32_t src;  /* first of its L+1 entries in the table of subspace offsets */
    uint32_t dst;  /* block-layout offset of its first slot with I = t = 0      */
    uint32_t blk;  /* block size: stride of the prefix cell I                   */
    uint32_t sub;  /* sub-block size: stride of t_c                             */
    uint32_t plen; /* pole size: stride of t_a                                  */
    uint8_t c, a;  /* levels of dims C and A                                    */
    uint8_t L;     /* last level of dim B                                       */
    uint8_t s;     /* level sum of dims 0..d-2: 2^s poles                       */
} sg_repack;

/* The repack table (nrows entries), the device offsets of the rows'
 * subspaces (S entries; both malloc'd) and the block sizes blk3[R] (3-D
 * block) and blk2[r] (sub-block) for every budget. */
int sg_layout_eval_tables(const sg_layout *L, sg_repack **repack, uint32_t **src, uint32_t *blk3, uint32_t *blk2);

#ifdef __cplusplus
}
#endif
#endif
