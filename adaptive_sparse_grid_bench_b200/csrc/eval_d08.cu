/* Evaluation kernels for d = 8 (see eval_impl.cuh); one dimension per file and
 * one kernel per SG_EVAL_PART so that they compile in parallel. */
#include "eval_impl.cuh"

#if SG_EVAL_PART == 0
template int eval_launch<8>(const EvalArgs *, void *);
#elif SG_EVAL_PART == 1
template int eval_batch_launch<8>(const EvalArgs *, const int2 *, int, void *);
#else
template int eval_shared_launch<8>(const EvalArgs *, const int2 *, int, const EvalArgs *, void *);
#endif
