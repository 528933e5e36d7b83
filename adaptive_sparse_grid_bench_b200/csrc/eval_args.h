/*
 * Arguments of the evaluation kernels and the per-dimension launchers
 * (instantiated in eval_d*.cu so that the kernels compile in parallel).
 */
#ifndef SG_EVAL_ARGS_H
#define SG_EVAL_ARGS_H

#include <stdint.h>

#include <vector_types.h>

#include "sg_kernels.h"

typedef sg_eval_args EvalArgs;

/* How much of the walk runs as fully unrolled code: 3-D blocks of budget <=
 * SG_EVAL_MAX_RF, leaf subtrees of the last prefix dim of budget <=
 * SG_EVAL_MAX_LEAF, of the last two prefix dims of budget <=
 * SG_EVAL_MAX_LEAF2.  d = 10, n = 10, 2^22 points at two points per thread: 156
 * ms with leaf budgets 3 and 2, 141.6 ms with 4 and 3, 137.4 ms with 5 and 3,
 * 135.0 ms with 5 and 4, whose gain is gone once small blocks load ahead
 * (eval_impl.cuh). */
#define SG_EVAL_MAX_RF 6
#define SG_EVAL_MAX_LEAF 5
#define SG_EVAL_MAX_LEAF2 3

/* Whole sums of one grid; whole sums of many grids of dimension D: items[b] =
 * (grid index into `grids` | share << 29, first point) for CTA b; sums shared
 * among warps, of many grids or of `one`. */
template <int D>
int eval_launch(const EvalArgs *A, void *stream);
template <int D>
int eval_batch_launch(const EvalArgs *grids, const int2 *items, int nitems, void *stream);
template <int D>
int eval_shared_launch(const EvalArgs *grids, const int2 *items, int nitems, const EvalArgs *one, void *stream);

#endif
