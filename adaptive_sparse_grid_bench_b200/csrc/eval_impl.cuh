/*
 * Evaluation kernels for sm_100a (instantiated per dimension in eval_d*.cu).
 *
 * Reference algorithm: evaluate0 in adaptive_sparse_grid_bench.c:1237-1274
 * (definition) and evaluate5 (c:1558-1688): for a query point x,
 *     u(x) = sum over subspaces l of  a[off(l) + idx(x, l)] * prod_k hat_k
 * with t_k = floor(x_k 2^l_k), idx(x, l) = row-major (t_0, ..., t_{d-1}) over
 * the subspace (dim 0 most significant) and hat_k = 1 - |x_k 2^(l_k+1) - (2t_k+1)|.
 *
 * B200 design.  One thread owns P query points; every warp walks the same
 * depth-first tree over the level vectors of the prefix dims 0..d-4 (each
 * dim's level ascending, sum(l) <= n-1, l_k <= limits[k]), so control flow is
 * uniform across the warp and partial products / partial cell indices are
 * shared by all subspaces below a node.  Below a prefix cell the walk reads
 * one block: every subspace of the three innermost dims (C = d-3, A = d-2,
 * B = d-1), stored contiguously in the block layout (sg_layout.h) with dim
 * B's levels of a row (c, a) folded into what a point needs of them: one
 * surplus (L = 0), a pair of surpluses (L = 1), or the value and slope of the
 * levels' piecewise linear sum on the point's half cell (L >= 2), at
 *     base + coff(c) + t_c sub(R-c) + aoff(a) + t_a plen(a) + 2 t_B:
 *   - blocks follow each other in walk order, so the block base is a running
 *     counter plus one multiply-add per point (no table);
 *   - a row of L+1 subspaces costs one address, one load (4 or 8 bytes) and
 *     one or two FMAs; the hats of dim B's levels 0 and 1 and the positions in
 *     the halves of levels 2..kYReg+1 are precomputed per point in registers
 *     (deeper rows, 10 % of the rows at d = 10, n = 10, compute theirs), the
 *     hats of dims A and C in this thread's column of shared memory;
 *   - the two points of a thread are computed with Blackwell's packed FP32x2
 *     instructions (FFMA2, FADD2, FMUL2 through __ffma2_rn, __fadd2_rn,
 *     __fmul2_rn): one instruction does both points' FMA, product or
 *     compensated add, with each point's rounding exactly as in scalar code,
 *     so results are bit-identical to one point per thread;
 *   - blocks of budget R <= kRFof<D> run fully unrolled; larger blocks
 *     loop over their planes and run each plane's 2-D sub-block fully
 *     unrolled behind a jump table.  A block or sub-block whose budget is within the limits of
 *     its dims has the regular shape whatever the limits, so limit-vector
 *     (adaptive) grids take the unrolled code too; a generic loop covers
 *     budgets above the limits, budgets >= kNB and d = 1;
 *   - most blocks sit under walk nodes of small remaining budget (at d=10,
 *     n=10, 8,008 of 11,440 blocks hold at most 4 subspaces), where loop and
 *     dispatch cost more than the gathers: the last prefix dim with budget
 *     <= kLeaf (levels and blocks) and the last two with budget <= kLeaf2 run
 *     as fully unrolled code with compile-time block sizes, in walk order, so
 *     results are bit-identical to the loop;
 *   - per prefix dim the walk keeps three values per point: the fractional
 *     part y = frac(x 2^l) (next level: doubling, exact in FP32), the cell
 *     index of the prefix (next level: 2*ix + bit) and the parent's product;
 *   - block sums of one prefix node are accumulated with FMAs and the node's
 *     total enters a Kahan-compensated accumulator.
 * Query points are put in spatial (Morton) order beforehand so the 32 points
 * of a warp share cells of the coarse subspaces and the gathers of a warp
 * touch few sectors; the grid is then served from L1/L2.
 */
#ifndef SG_EVAL_IMPL_CUH
#define SG_EVAL_IMPL_CUH

#include <cuda_runtime.h>
#include <stdint.h>

#include "eval_args.h"

namespace sgeval {

constexpr int kThreads = 256;
constexpr int kNB = 10; /* 2-D sub-blocks of budget r < kNB run fully unrolled */
constexpr int kRF = SG_EVAL_MAX_RF; /* 3-D blocks of budget R <= kRF can run unrolled */
static_assert(kRF == 6, "block_sum's jump table covers budgets 0..6");
/* largest budget of an unrolled 3-D block (above 12 dims, where the walk's own
 * state is larger, blocks of budget 6 only add spills) */
template <int D>
constexpr int kRFof = D <= 12 ? kRF : 5;
constexpr int kTB = 15; /* T = floor(x 2^15) holds the cells of levels 0..15   */
constexpr int kYReg = 1; /* positions in the halves of levels 2..kYReg+1 sit in registers */

/* P = 2 floats, one per point of a thread: packed FP32x2 instructions. */
template <int P>
struct FV;
template <>
struct FV<2> {
    float2 v;
    __device__ __forceinline__ float get(int p) const { return p ? v.y : v.x; }
    __device__ __forceinline__ void set(int p, float x)
    {
        if (p) v.y = x;
        else v.x = x;
    }
    static __device__ __forceinline__ FV all(float x) { return FV{make_float2(x, x)}; }
};
__device__ __forceinline__ FV<2> vfma(FV<2> a, FV<2> b, FV<2> c) { return FV<2>{__ffma2_rn(a.v, b.v, c.v)}; }
__device__ __forceinline__ FV<2> vmul(FV<2> a, FV<2> b) { return FV<2>{__fmul2_rn(a.v, b.v)}; }
__device__ __forceinline__ FV<2> vadd(FV<2> a, FV<2> b) { return FV<2>{__fadd2_rn(a.v, b.v)}; }
__device__ __forceinline__ FV<2> vsub(FV<2> a, FV<2> b)
{
    return FV<2>{__fadd2_rn(a.v, make_float2(-b.v.x, -b.v.y))};
}

/* compensated (Kahan) s += v, c holding the running rounding error */
template <int P>
__device__ __forceinline__ void kahan_add(FV<P> &s, FV<P> &c, FV<P> v)
{
    const FV<P> y = vsub(v, c);
    const FV<P> t = vadd(s, y);
    c = vsub(vsub(t, s), y);
    s = t;
}

/* cell index at level l (0..15) from T = floor(x 2^15): T >> (15 - l).
 * Level 0 has one cell and T < 2^15 for every x in [0,1) (x 2^15 is exact),
 * so its index is 0; that is written out as a constant because the compiler
 * cannot bound T, which comes from a float conversion, and would otherwise
 * shift and multiply a zero in every row and plane of level 0. */
__device__ __forceinline__ uint32_t cell_at(uint32_t T, int l) { return l == 0 ? 0u : T >> (kTB - l); }

/* hat at the current level from the fractional part y = frac(x 2^l) */
__device__ __forceinline__ float hat_of(float y) { return 1.0f - fabsf(fmaf(2.0f, y, -1.0f)); }

/* next level: y <- frac(2y) (exact), returns floor(2y) */
__device__ __forceinline__ uint32_t step_y(float &y)
{
    const float y2 = y + y;
    const bool b = y2 >= 1.0f;
    y = b ? y2 - 1.0f : y2;
    return (uint32_t)b;
}

template <int P>
__device__ __forceinline__ FV<P> hats(const FV<P> &y)
{
    FV<P> h;
#pragma unroll
    for (int p = 0; p < P; ++p) h.set(p, hat_of(y.get(p)));
    return h;
}

/* The walk's view of arguments that sit in shared memory: the scalars it
 * uses everywhere in registers, the tables read in place. */
struct GridView {
    const float *alpha;
    int nm1, lim2, lim3;
    const int *lim;
    const uint32_t *blk3, *blk2, *seg;
    __device__ __forceinline__ explicit GridView(const EvalArgs &A)
        : alpha(A.alpha), nm1(A.nm1), lim2(A.lim2), lim3(A.lim3), lim(A.lim), blk3(A.blk3), blk2(A.blk2), seg(A.seg)
    {
    }
};

/* A hat from this thread's column of shared memory.  Written as assembly so
 * that the compiler does not look for the thousands of possibly equal loads of
 * the unrolled blocks (which took minutes per kernel) nor keeps their values in
 * registers across blocks; a block reads each hat it needs once.  The columns
 * are written once, before a compiler barrier, and only read after it. */
template <int P>
__device__ __forceinline__ FV<P> lds_hat(uint32_t column, int slot)
{
    static_assert(P == 2, "two points per thread");
    FV<P> h;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];"
                 : "=f"(h.v.x), "=f"(h.v.y)
                 : "r"(column + (uint32_t)slot * (uint32_t)(kThreads * sizeof(FV<P>))));
    return h;
}

/* Per-point values of the three innermost dims. */
template <int P>
struct Inner {
    FV<P> hB[2];          /* hat of dim B at levels 0, 1             */
    FV<P> yB[kYReg > 0 ? kYReg : 1]; /* frac(x_B 2^(L+1)), L = 2 ..       */
    FV<P> xB;
    uint32_t TB[P];       /* floor(x_B 2^15): cells and halves of dim B */
    uint32_t sh;          /* shared address of this thread's hats of dims A, C */
    uint32_t TA[P];       /* floor(x_A 2^15): t_a = TA >> (15 - a)   */
    uint32_t TC[P];       /* floor(x_C 2^15)                         */
    __device__ __forceinline__ FV<P> hA(int a) const { return lds_hat<P>(sh, a); }
    /* position in the half of a cell of level L >= 2: frac(x_B 2^(L+1)),
     * exact (the scaling and the difference are) */
    __device__ __forceinline__ FV<P> y(int L) const
    {
        if (L - 2 < kYReg) return yB[L - 2];
        const FV<P> t = vmul(xB, FV<P>::all((float)(2u << L)));
        FV<P> f;
#pragma unroll
        for (int p = 0; p < P; ++p) f.set(p, truncf(t.get(p)));
        return vsub(t, f);
    }
    __device__ __forceinline__ FV<P> hC(int c) const { return lds_hat<P>(sh, kNB + c); }
};
constexpr int kHatSlots = kNB + kRF + 1;

/* Regular shapes: blocks whose budget is within the innermost limits. */
__host__ __device__ constexpr uint32_t plen_reg(int r, int a) { return SG_POLE_SLOTS(r - a); }
__host__ __device__ constexpr uint32_t aoff_reg(int r, int a)
{
    uint32_t o = 0;
    for (int q = 0; q < a; ++q) o += (1u << q) * plen_reg(r, q);
    return o;
}
__host__ __device__ constexpr uint32_t blk2_reg(int r) { return aoff_reg(r, r + 1); }
__host__ __device__ constexpr uint32_t coff_reg(int R, int c)
{
    uint32_t o = 0;
    for (int q = 0; q < c; ++q) o += (1u << q) * blk2_reg(R - q);
    return o;
}

/* A row of dim B with last level L, in two parts so that a block's loads can
 * all be in flight before its first sum: what the point needs of the row at
 * `at` (one load, sg_layout.h), and from it the sum over the row's levels of
 * surplus * hat. */
template <int P>
struct RowData {
    float2 w[P]; /* L = 0: .x only */
};
template <int L, int P>
__device__ __forceinline__ void row_load(const float *__restrict__ alpha, const uint32_t (&at)[P], const Inner<P> &in,
                                         RowData<P> &d)
{
#pragma unroll
    for (int p = 0; p < P; ++p) {
        if constexpr (L == 0)
            d.w[p].x = __ldg(alpha + at[p]);
        else
            d.w[p] = __ldg(reinterpret_cast<const float2 *>(
                alpha + (at[p] + 2 * cell_at(in.TB[p], L == 1 ? 1 : L + 1))));
    }
}
template <int L, int P>
__device__ __forceinline__ FV<P> row_sum(const RowData<P> &d, const Inner<P> &in)
{
    FV<P> v0, v1;
#pragma unroll
    for (int p = 0; p < P; ++p) {
        v0.set(p, d.w[p].x);
        if constexpr (L > 0) v1.set(p, d.w[p].y);
    }
    if constexpr (L == 0) return vmul(in.hB[0], v0);
    else if constexpr (L == 1) return vfma(in.hB[1], v1, vmul(in.hB[0], v0));
    else return vfma(in.y(L), v1, v0);
}

/* address of this point's pole in row a of a sub-block of budget r */
template <int r, int a, int P>
__device__ __forceinline__ void row_at(const uint32_t (&base)[P], const Inner<P> &in, uint32_t (&at)[P])
{
#pragma unroll
    for (int p = 0; p < P; ++p) at[p] = base[p] + aoff_reg(r, a) + cell_at(in.TA[p], a) * plen_reg(r, a);
}
/* address of this point's sub-block in plane c of a block of budget R */
template <int R, int c, int P>
__device__ __forceinline__ void plane_at(const uint32_t (&base)[P], const Inner<P> &in, uint32_t (&sb)[P])
{
#pragma unroll
    for (int p = 0; p < P; ++p) sb[p] = base[p] + coff_reg(R, c) + cell_at(in.TC[p], c) * blk2_reg(R - c);
}

/* 2-D sub-block of budget r: rows a = 0..r, row a holds 2^a poles of r-a+1
 * levels.  s = sum_a hA[a] * (row sum). */
template <int r, int a, int P, int NA>
__device__ __forceinline__ void block2_fixed(const float *__restrict__ alpha, const uint32_t (&base)[P],
                                             const Inner<P> &in, const FV<P> (&hA)[NA], FV<P> &s)
{
    uint32_t at[P];
    RowData<P> d;
    row_at<r, a, P>(base, in, at);
    row_load<r - a, P>(alpha, at, in, d);
    const FV<P> sr = row_sum<r - a, P>(d, in);
    s = (a == 0) ? vmul(hA[0], sr) : vfma(hA[a], sr, s);
    if constexpr (a < r) block2_fixed<r, a + 1, P, NA>(alpha, base, in, hA, s);
}

/* planes C..R of a fully unrolled 3-D block of budget R */
template <int R, int C, int P, int NA>
__device__ __forceinline__ void block3_planes(const float *__restrict__ alpha, const uint32_t (&base)[P],
                                              const Inner<P> &in, const FV<P> (&hA)[NA], FV<P> &s)
{
    uint32_t sb[P];
    FV<P> s2;
    plane_at<R, C, P>(base, in, sb);
    block2_fixed<R - C, 0, P, NA>(alpha, sb, in, hA, s2);
    s = (C == 0) ? vmul(in.hC(0), s2) : vfma(in.hC(C), s2, s);
    if constexpr (C < R) block3_planes<R, C + 1, P, NA>(alpha, base, in, hA, s);
}

/* Small blocks in two passes, every row loaded before the first is summed
 * (in the order of block3_planes, so the results are the same bits).  The
 * walk is bound by the latency of its gathers at 16 warps per SM; with the
 * sums in between, ptxas keeps few loads in flight.  d = 10, n = 10, 2^22
 * points, two points per thread: 137.4 ms without, 128.8 ms for blocks of
 * budget <= 3 (10 rows), 141.4 ms for <= 4 (15 rows: the registers run out). */
template <int P>
constexpr int kAhead = 3;
template <int R, int c, int a, int i, int P, int N>
__device__ __forceinline__ void block3_load(const float *__restrict__ alpha, const uint32_t (&base)[P],
                                            const Inner<P> &in, RowData<P> (&d)[N])
{
    uint32_t sb[P], at[P];
    plane_at<R, c, P>(base, in, sb);
    row_at<R - c, a, P>(sb, in, at);
    row_load<R - c - a, P>(alpha, at, in, d[i]);
    if constexpr (a < R - c) block3_load<R, c, a + 1, i + 1, P, N>(alpha, base, in, d);
    else if constexpr (c < R) block3_load<R, c + 1, 0, i + 1, P, N>(alpha, base, in, d);
}
template <int R, int c, int a, int i, int P, int N>
__device__ __forceinline__ void block3_sum(const Inner<P> &in, const RowData<P> (&d)[N], const FV<P> (&hA)[R + 1],
                                           FV<P> &s2, FV<P> &s)
{
    const FV<P> sr = row_sum<R - c - a, P>(d[i], in);
    s2 = (a == 0) ? vmul(hA[0], sr) : vfma(hA[a], sr, s2);
    if constexpr (a < R - c) {
        block3_sum<R, c, a + 1, i + 1, P, N>(in, d, hA, s2, s);
    } else {
        s = (c == 0) ? vmul(in.hC(0), s2) : vfma(in.hC(c), s2, s);
        if constexpr (c < R) block3_sum<R, c + 1, 0, i + 1, P, N>(in, d, hA, s2, s);
    }
}

/* The cells behind a compiler barrier, per block: every address term made of
 * them is the same for the whole walk, and hoisted out of its loops the terms of
 * the unrolled blocks take registers from the loads.  d = 10, n = 6, 2^20 points:
 * 1851 -> 1779 us; n = 10, 2^22 points: 136.7 -> 135.3 ms. */
template <int P>
__device__ __forceinline__ Inner<P> here(const Inner<P> &in)
{
    Inner<P> o = in;
#pragma unroll
    for (int p = 0; p < P; ++p) asm volatile("" : "+r"(o.TA[p]), "+r"(o.TB[p]), "+r"(o.TC[p]));
    return o;
}

/* Fully unrolled 3-D block of budget R. */
template <int R, int P>
__device__ __forceinline__ void block3_fixed(const float *__restrict__ alpha, const uint32_t (&base)[P],
                                             const Inner<P> &inner, FV<P> &s)
{
        const Inner<P> in = here(inner);
    FV<P> hA[R + 1];
#pragma unroll
    for (int a = 0; a <= R; ++a) hA[a] = in.hA(a);
    if constexpr (R <= kAhead<P>) {
        constexpr int N = (R + 1) * (R + 2) / 2;
        RowData<P> d[N];
        FV<P> s2;
        block3_load<R, 0, 0, 0, P, N>(alpha, base, in, d);
        block3_sum<R, 0, 0, 0, P, N>(in, d, hA, s2, s);
    } else {
        block3_planes<R, 0, P, R + 1>(alpha, base, in, hA, s);
    }
}

/* Generic sub-block of budget r (limits, r >= kNB): runtime loops. */
template <int P>
__device__ __forceinline__ void block2_generic(const float *__restrict__ alpha, int r, int limA, int limB,
                                               const float (&xA)[P], const float (&xB)[P], bool hasA,
                                               const uint32_t (&base)[P], FV<P> &s)
{
    const int amax = min(r, limA);
    uint32_t aoff = 0;
    FV<P> yA;
    uint32_t tA[P];
#pragma unroll
    for (int p = 0; p < P; ++p) {
        yA.set(p, xA[p]);
        tA[p] = 0;
    }
    s = FV<P>::all(0.0f);
    for (int a = 0; a <= amax; ++a) {
        if (a) {
#pragma unroll
            for (int p = 0; p < P; ++p) {
                float y = yA.get(p);
                tA[p] = 2 * tA[p] + step_y(y);
                yA.set(p, y);
            }
        }
        const int L = min(r - a, limB);
        const uint32_t plen = SG_POLE_SLOTS(L);
        FV<P> sr;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const float *pole = alpha + (base[p] + aoff + tA[p] * plen);
            if (L == 0) {
                sr.set(p, __fmul_rn(hat_of(xB[p]), __ldg(pole)));
            } else {
                /* cell of level 1, or half of a cell of level L, and the
                 * position in it (exact) */
                const float t = xB[p] * (float)(L == 1 ? 2u : 2u << L), f = truncf(t), y = t - f;
                const float2 w = __ldg(reinterpret_cast<const float2 *>(pole + 2 * (uint32_t)f));
                sr.set(p, L == 1 ? fmaf(hat_of(y), w.y, __fmul_rn(hat_of(xB[p]), w.x)) : fmaf(y, w.y, w.x));
            }
        }
        s = vfma(hasA ? hats(yA) : FV<P>::all(1.0f), sr, s);
        aoff += (1u << a) * plen;
    }
}

/* Sub-block of budget r: unrolled (r within the limits, r < kNB) or generic. */
template <int D, int P, typename GA>
__device__ __forceinline__ void block2_any(const GA &A, int r, const Inner<P> &in, const float (&xA)[P],
                                           const float (&xB)[P], const uint32_t (&base)[P], FV<P> &s)
{
    if (D >= 2 && r <= A.lim2) {
        switch (r) {
#define SG_BLK2(RR)                                                          \
    case RR: {                                                               \
        FV<P> hA[RR + 1];                                                    \
        _Pragma("unroll") for (int a = 0; a <= RR; ++a) hA[a] = in.hA(a);    \
        block2_fixed<RR, 0, P, RR + 1>(A.alpha, base, here(in), hA, s);      \
        return;                                                              \
    }
            SG_BLK2(0) SG_BLK2(1) SG_BLK2(2) SG_BLK2(3) SG_BLK2(4)
            SG_BLK2(5) SG_BLK2(6) SG_BLK2(7) SG_BLK2(8) SG_BLK2(9)
#undef SG_BLK2
        default: break;
        }
    }
    block2_generic<P>(A.alpha, r, D >= 2 ? A.lim[D >= 2 ? D - 2 : 0] : 0, A.lim[D - 1], xA, xB, D >= 2, base, s);
}

/* Sum over the block of budget R at `base` for every point. */
template <int D, int P, typename GA>
__device__ __forceinline__ void block_sum(const GA &A, int R, const Inner<P> &in, const float (&xC)[P],
                                          const float (&xA)[P], const float (&xB)[P], const uint32_t (&base)[P],
                                          FV<P> &s)
{
    if constexpr (D >= 3) {
        if (R <= kRFof<D> && R <= A.lim3) {
            switch (R) {
            case 0: block3_fixed<0, P>(A.alpha, base, in, s); return;
            case 1: block3_fixed<1, P>(A.alpha, base, in, s); return;
            case 2: block3_fixed<2, P>(A.alpha, base, in, s); return;
            case 3: block3_fixed<3, P>(A.alpha, base, in, s); return;
            case 4: block3_fixed<4, P>(A.alpha, base, in, s); return;
            case 5:
                if constexpr (kRFof<D> > 5) {
                    block3_fixed<5, P>(A.alpha, base, in, s);
                    return;
                }
                [[fallthrough]];
            default: block3_fixed<kRFof<D>, P>(A.alpha, base, in, s); return;
            }
        }
    }
    /* plane loop; dim C is absent (limit 0) for d < 3 */
    const int cmax = D >= 3 ? min(R, A.lim[D >= 3 ? D - 3 : 0]) : 0;
    uint32_t coff = 0;
    FV<P> yC;
    uint32_t tC[P];
#pragma unroll
    for (int p = 0; p < P; ++p) {
        yC.set(p, xC[p]);
        tC[p] = 0;
    }
    s = FV<P>::all(0.0f);
    for (int c = 0; c <= cmax; ++c) {
        if (c) {
#pragma unroll
            for (int p = 0; p < P; ++p) {
                float y = yC.get(p);
                tC[p] = 2 * tC[p] + step_y(y);
                yC.set(p, y);
            }
        }
        const uint32_t sub = A.blk2[R - c];
        uint32_t sb[P];
        FV<P> s2;
#pragma unroll
        for (int p = 0; p < P; ++p) sb[p] = base[p] + coff + tC[p] * sub;
        block2_any<D, P>(A, R - c, in, xA, xB, sb, s2);
        s = vfma(D >= 3 ? hats(yC) : FV<P>::all(1.0f), s2, s);
        coff += (1u << c) * sub;
    }
}

/* level state (y, cell index, parent product) of the upper prefix dims
 * K < kUpper (K <= D-6, at most 7 of them so that two CTAs still fit an SM
 * at d = 20), kept in shared memory while the subtree below runs */
template <int D>
constexpr int kUpper = D >= 6 ? (D - 5 < 7 ? D - 5 : 7) : 0;

/* Segments of the sum (sg_layout.h), as block-layout offsets compared with
 * the walk's running offset `cur`.  The walk has no registers to spare, so it
 * carries only the end of the current segment and the start of the warp's
 * range (several warps may share a sum); the rest lives in local memory and is touched once per segment by a function that
 * is not inlined (inlined, its registers cost 9 % at d = 10, n = 10). */
struct Range {
    uint32_t next; /* end of the current segment, 0xFFFFFFFF: none follows   */
    uint32_t lo;   /* first offset of the warp's range, 0xFFFFFFFF: all done */
};
template <int P>
struct Tail {
    const uint32_t *bounds;
    int s, end, nseg, emit;           /* current segment, end of the warp's own */
    float part[2][P], total[2][P];    /* compensated sums                       */
    float *out[P];                    /* shared sums: the points in part_out, or NULL */
    int64_t stride;
    bool valid[P], nan_in[P];
};

/* adds the compensated sum (vs, vc) to acc, its compensation included: a segment
 * rounded to one float where it ends would cost up to 5 % in the error of the
 * total */
template <int P>
__device__ __forceinline__ void fold(float (&acc)[2][P], FV<P> vs, FV<P> vc)
{
    FV<P> s, c;
#pragma unroll
    for (int p = 0; p < P; ++p) {
        s.set(p, acc[0][p]);
        c.set(p, acc[1][p]);
    }
    kahan_add(s, c, vs);
    kahan_add(s, c, vsub(FV<P>::all(0.0f), vc));
#pragma unroll
    for (int p = 0; p < P; ++p) {
        acc[0][p] = s.get(p);
        acc[1][p] = c.get(p);
    }
}

/* moves the compensated sum in acc out */
template <int P>
__device__ __forceinline__ void take(float (&acc)[2][P], FV<P> &s, FV<P> &c)
{
#pragma unroll
    for (int p = 0; p < P; ++p) {
        s.set(p, acc[0][p]);
        c.set(p, acc[1][p]);
        acc[0][p] = acc[1][p] = 0.0f;
    }
}

/* Ends the current segment, whose compensated sum is (v, c); returns the next
 * segment's end. */
template <int P>
__device__ __noinline__ uint32_t close_segment(Tail<P> *t, FV<P> v, FV<P> c)
{
    const int s = t->s++;
    int k = s;
    bool whole = true;
    if (t->emit != SG_EMIT_SEGS) {
        fold<P>(t->part, v, c);
        whole = (s + 1) % SG_SEG_PER_PART == 0 || s + 1 == t->nseg;
        if (whole) {
            take<P>(t->part, v, c);
            k = s / SG_SEG_PER_PART;
            if (t->emit == SG_EMIT_SUM) fold<P>(t->total, v, c);
        }
    }
    if (whole && t->emit != SG_EMIT_SUM) {
#pragma unroll
        for (int p = 0; p < P; ++p)
            if (t->out[p]) {
                t->out[p][2 * k * t->stride] =
                    t->valid[p] ? v.get(p) : (t->nan_in[p] ? __int_as_float(0x7fc00000) : 0.0f);
                t->out[p][(2 * k + 1) * t->stride] = t->valid[p] ? c.get(p) : 0.0f;
            }
    }
    return s + 2 < t->nseg ? __ldg(t->bounds + s + 2) : 0xFFFFFFFFu;
}

/* Largest budgets of the unrolled subtrees of the last prefix dim (kLeaf) and of
 * the last two (kLeaf2).  Above 12 dims the walk's own loops take most of the
 * time and the small subtrees most of the gain, while the unrolled code takes
 * ptxas four to ten times as long with the budgets of the lower dims.  Whole sums
 * with loops only / these budgets / 5 and 3: d = 13, n = 6, 5e5 points 7.43 /
 * 4.39 / 3.99 ms, d = 16, n = 5, 3e5 points 3.17 / 2.18 / 2.34 ms. */
template <int D>
constexpr int kLeaf = D <= 12 ? SG_EVAL_MAX_LEAF : 2;
template <int D>
constexpr int kLeaf2 = D <= 12 ? SG_EVAL_MAX_LEAF2 : 1;
static_assert(SG_EVAL_MAX_LEAF2 == SG_SEG_UNIT_BUDGET, "segments start outside the unrolled subtrees");
static_assert(SG_EVAL_MAX_LEAF <= 5 && SG_EVAL_MAX_LEAF2 <= 3,
              "the walk's jump tables cover leaf budgets 0..5 and 0..3");

/* next level of one prefix dim for every point: y doubles, the cell index
 * takes the next bit */
template <int P>
__device__ __forceinline__ void step_all(FV<P> &y, uint32_t (&ix)[P])
{
#pragma unroll
    for (int p = 0; p < P; ++p) {
        float t = y.get(p);
        ix[p] = 2 * ix[p] + step_y(t);
        y.set(p, t);
    }
}

/* Levels l = L..B of the last prefix dim and their 3-D blocks of budget
 * B - l, fully unrolled (every shape regular: B within the limits). */
template <int D, int P, int B, int L, typename GA>
__device__ __forceinline__ void leaf_group(const GA &A, uint32_t &cur, const Inner<P> &in, const FV<P> &pin,
                                           FV<P> &y, uint32_t (&ix)[P], FV<P> &acc)
{
    if constexpr (L > 0) step_all<P>(y, ix);
    constexpr int R = B - L;
    constexpr uint32_t blk = coff_reg(R, R + 1);
    uint32_t base[P];
    FV<P> s;
#pragma unroll
    for (int p = 0; p < P; ++p) base[p] = cur + ix[p] * blk;
    cur += blk << (A.nm1 - R);
    block3_fixed<R, P>(A.alpha, base, in, s);
    acc = vfma(vmul(pin, hats(y)), s, acc);
    if constexpr (L < B) leaf_group<D, P, B, L + 1>(A, cur, in, pin, y, ix, acc);
}

/* the coordinates of prefix dim K of this thread's points */
template <int P>
__device__ __forceinline__ FV<P> load_y(const float *sx, int K, int tid)
{
    FV<P> y;
#pragma unroll
    for (int p = 0; p < P; ++p) y.set(p, sx[(K * P + p) * kThreads + tid]);
    return y;
}

/* Levels l = L..B of prefix dim K = D-5, each followed by the unrolled
 * leaf group of dim D-4 with budget B - l (one compensated add per group,
 * as in the walk). */
template <int D, int K, int P, int B, int L, typename GA>
__device__ __forceinline__ void leaf_group2(const GA &A, const float *sx, int tid, uint32_t &cur,
                                            const Inner<P> &in, const FV<P> &pin, FV<P> &y, uint32_t (&ix)[P],
                                            FV<P> &sum, FV<P> &comp)
{
    if constexpr (L > 0) step_all<P>(y, ix);
    const FV<P> pn = vmul(pin, hats(y));
    FV<P> y2 = load_y<P>(sx, K + 1, tid);
    FV<P> acc = FV<P>::all(0.0f);
    uint32_t ix2[P];
#pragma unroll
    for (int p = 0; p < P; ++p) ix2[p] = ix[p];
    leaf_group<D, P, B - L, 0>(A, cur, in, pn, y2, ix2, acc);
    kahan_add(sum, comp, acc);
    if constexpr (L < B) leaf_group2<D, K, P, B, L + 1>(A, sx, tid, cur, in, pin, y, ix, sum, comp);
}

/* Walk over prefix dim K (K <= D-4); children of depth D-4 are blocks.
 * Segments start at iterations of the loops at depth K <= D-5 (D = 4: of its
 * only loop), so subtrees outside the warp's range are skipped there by their
 * extents, and segments are closed where the innermost of those loops
 * starts an iteration (every outer iteration starts one of it). */
template <int D, int K, int P, bool SH>
struct Walk {
    static constexpr bool kLoop = D == 4 ? K == 0 : K + 5 <= D;  /* may skip  */
    static constexpr bool kClose = D == 4 ? K == 0 : K + 5 == D; /* closes    */

    /* child of budget `left` lies before the range (or the range is done):
     * step over it */
    template <typename GA>
    static __device__ __forceinline__ bool skip(const GA &A, const Range &rg, int left, uint32_t &cur)
    {
        if constexpr (kLoop && SH) {
            if (cur < rg.lo) {
                const uint32_t ext = __ldg(A.seg + (K + 1) * (A.nm1 + 1) + left);
                if (cur + ext <= rg.lo) {
                    cur += ext;
                    return true;
                }
            }
        }
        return false;
    }
    /* closes the segments that end at or before cur; true when the warp's
     * own are all closed */
    static __device__ __forceinline__ bool close(Range &rg, Tail<P> *tl, uint32_t cur, FV<P> &sum, FV<P> &comp)
    {
        while (cur >= rg.next) {
            rg.next = close_segment<P>(tl, sum, comp);
            sum = comp = FV<P>::all(0.0f);
            if constexpr (SH) {
                if (tl->s >= tl->end) {
                    rg.lo = rg.next = 0xFFFFFFFFu;
                    return true;
                }
            }
        }
        return false;
    }

    template <typename GA>
    static __device__ __forceinline__ void run(const GA &A, const float *sx, int tid, int budget,
                                               uint32_t &cur, Range &rg, Tail<P> *tl, const Inner<P> &in,
                                               const float (&xC)[P],
                                               const float (&xA)[P], const float (&xB)[P], const FV<P> &pin,
                                               const uint32_t (&ixin)[P], FV<P> &sum, FV<P> &comp)
    {
        if constexpr (K + 6 <= D && K < kUpper<D>) {
            /* upper prefix dim: its level state lives in this thread's
             * shared-memory slots while the subtree below runs, so it holds
             * no registers there */
            constexpr int NPX = D >= 4 ? D - 3 : 1;
            volatile float *ws = const_cast<float *>(sx) + NPX * P * kThreads + (K * 3 * P) * kThreads + tid;
            const int lmax = min(A.lim[K], budget);
#pragma unroll
            for (int p = 0; p < P; ++p) {
                ws[(0 * P + p) * kThreads] = sx[(K * P + p) * kThreads + tid];
                ws[(1 * P + p) * kThreads] = __uint_as_float(ixin[p]);
                ws[(2 * P + p) * kThreads] = pin.get(p);
            }
#pragma unroll 1
            for (int l = 0; l <= lmax; ++l) {
                FV<P> y, pp, yn;
                uint32_t ix[P], ixn[P];
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    y.set(p, ws[(0 * P + p) * kThreads]);
                    ix[p] = ixn[p] = __float_as_uint(ws[(1 * P + p) * kThreads]);
                    pp.set(p, ws[(2 * P + p) * kThreads]);
                }
                /* the next level's state */
                yn = y;
                step_all<P>(yn, ixn);
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    ws[(0 * P + p) * kThreads] = yn.get(p);
                    ws[(1 * P + p) * kThreads] = __uint_as_float(ixn[p]);
                }
                if (skip(A, rg, budget - l, cur)) continue;
                const FV<P> pn = vmul(pp, hats(y));
                Walk<D, K + 1, P, SH>::run(A, sx, tid, budget - l, cur, rg, tl, in, xC, xA, xB, pn, ix, sum, comp);
            }
            return;
        }
        if constexpr (kClose && D > 4) {
            /* the first iteration's close, before the unrolled forms below */
            if (close(rg, tl, cur, sum, comp)) return;
        }
        const int lmax = min(A.lim[K], budget);
        FV<P> y = load_y<P>(sx, K, tid);
        FV<P> acc = FV<P>::all(0.0f);
        uint32_t ix[P];
#pragma unroll
        for (int p = 0; p < P; ++p) ix[p] = ixin[p];
        if constexpr (K + 1 == D - 4) {
            if (budget <= kLeaf2<D> && budget <= A.lim[K] && budget <= A.lim[K + 1] && budget <= A.lim3) {
                switch (budget) {
                case 0: leaf_group2<D, K, P, 0, 0>(A, sx, tid, cur, in, pin, y, ix, sum, comp); break;
                case 1: leaf_group2<D, K, P, 1, 0>(A, sx, tid, cur, in, pin, y, ix, sum, comp); break;
                case 2:
                    if constexpr (kLeaf2<D> >= 2) leaf_group2<D, K, P, 2, 0>(A, sx, tid, cur, in, pin, y, ix, sum, comp);
                    break;
                case 3:
                    if constexpr (kLeaf2<D> >= 3) leaf_group2<D, K, P, 3, 0>(A, sx, tid, cur, in, pin, y, ix, sum, comp);
                    break;
                default: break;
                }
                return;
            }
        }
        if constexpr (K == D - 4) {
            if (budget <= kLeaf<D> && budget <= A.lim[K] && budget <= A.lim3) {
                switch (budget) {
                case 0: leaf_group<D, P, 0, 0>(A, cur, in, pin, y, ix, acc); break;
                case 1: leaf_group<D, P, 1, 0>(A, cur, in, pin, y, ix, acc); break;
                case 2: leaf_group<D, P, 2, 0>(A, cur, in, pin, y, ix, acc); break;
                case 3:
                    if constexpr (kLeaf<D> >= 3) leaf_group<D, P, 3, 0>(A, cur, in, pin, y, ix, acc);
                    break;
                case 4:
                    if constexpr (kLeaf<D> >= 4) leaf_group<D, P, 4, 0>(A, cur, in, pin, y, ix, acc);
                    break;
                case 5:
                    if constexpr (kLeaf<D> >= 5) leaf_group<D, P, 5, 0>(A, cur, in, pin, y, ix, acc);
                    break;
                default: break;
                }
                kahan_add(sum, comp, acc);
                return;
            }
        }
#pragma unroll 1
        for (int l = 0; l <= lmax; ++l, step_all<P>(y, ix)) {
            if (skip(A, rg, budget - l, cur)) continue;
            if constexpr (kClose) {
                if constexpr (D == 4) {
                    if (cur >= rg.next) {
                        kahan_add(sum, comp, acc);
                        acc = FV<P>::all(0.0f);
                    }
                }
                if (close(rg, tl, cur, sum, comp)) return;
            }
            const FV<P> pn = vmul(pin, hats(y));
            if constexpr (K == D - 4) {
                const int R = budget - l;
                const uint32_t blk = A.blk3[R];
                uint32_t base[P];
                FV<P> s;
#pragma unroll
                for (int p = 0; p < P; ++p) base[p] = cur + ix[p] * blk;
                cur += blk << (A.nm1 - R);
                block_sum<D, P>(A, R, in, xC, xA, xB, base, s);
                acc = vfma(pn, s, acc);
            } else {
                Walk<D, K + 1, P, SH>::run(A, sx, tid, budget - l, cur, rg, tl, in, xC, xA, xB, pn, ix, sum, comp);
            }
        }
        if constexpr (K == D - 4) kahan_add(sum, comp, acc);
    }
};

/* Evaluates this thread's points first, first + 32, ..., first + 32(P-1)
 * (those below `end`) against grid A; sx is this CTA's shared coordinate
 * buffer, shat its shared hats of dims A and C; share = which of the
 * A.nshare shares of the segments this warp adds up. */
template <int D, int P, bool SH, typename GA>
__device__ __forceinline__ void eval_points(const EvalArgs &A, const GA &G, float *sx, FV<P> *shat, int tid, int64_t first,
                                            int64_t end, int share)
{
    float xC[P], xA[P], xB[P];
    bool valid[P], nan_in[P];
#pragma unroll
    for (int p = 0; p < P; ++p) {
        const int64_t i = first + 32 * p;
        float x[D];
        valid[p] = i < end;
        nan_in[p] = false;
        bool inside = true;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const float v = valid[p] ? A.coords[i * D + k] : 0.0f;
            nan_in[p] |= (v != v);
            inside &= (v >= 0.0f) && (v < 1.0f);
            x[k] = v;
        }
        /* outside [0,1)^d every basis function is 0: walk at x = 0 (always
         * in range) and write 0 (NaN for NaN input) instead */
        if (!inside) {
#pragma unroll
            for (int k = 0; k < D; ++k) x[k] = 0.0f;
        }
        valid[p] = valid[p] && inside;
#pragma unroll
        for (int k = 0; k + 3 < D; ++k) sx[(k * P + p) * kThreads + tid] = x[k];
        xC[p] = D >= 3 ? x[D >= 3 ? D - 3 : 0] : 0.0f;
        xA[p] = D >= 2 ? x[D >= 2 ? D - 2 : 0] : 0.0f;
        xB[p] = x[D - 1];
    }

    Inner<P> in;
    in.sh = (uint32_t)__cvta_generic_to_shared(shat + tid);
    FV<P> *const shw = shat + tid;
#pragma unroll
    for (int p = 0; p < P; ++p) {
        float y = xB[p];
        in.xB.set(p, y);
        in.hB[0].set(p, hat_of(y));
        (void)step_y(y);
        in.hB[1].set(p, hat_of(y));
        (void)step_y(y);
#pragma unroll
        for (int j = 0; j < kYReg; ++j) {
            (void)step_y(y);
            in.yB[j].set(p, y);
        }
        in.TB[p] = (uint32_t)(xB[p] * (float)(1u << kTB));
        in.TA[p] = (uint32_t)(xA[p] * (float)(1u << kTB));
        in.TC[p] = (uint32_t)(xC[p] * (float)(1u << kTB));
    }
    {
        FV<P> yA, yC;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            yA.set(p, xA[p]);
            yC.set(p, xC[p]);
        }
#pragma unroll
        for (int j = 0; j < kNB; ++j) {
            if (j)
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    float y = yA.get(p);
                    (void)step_y(y);
                    yA.set(p, y);
                }
            shw[j * kThreads] = hats(yA);
        }
#pragma unroll
        for (int j = 0; j <= kRF; ++j) {
            if (j)
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    float y = yC.get(p);
                    (void)step_y(y);
                    yC.set(p, y);
                }
            shw[(kNB + j) * kThreads] = hats(yC);
        }
    }

    asm volatile("" ::: "memory"); /* the hats are stored before lds_hat reads them */

    FV<P> sum = FV<P>::all(0.0f), comp = FV<P>::all(0.0f);
    uint32_t cur = 0;
    if constexpr (D >= 4) {
        const FV<P> pin = FV<P>::all(1.0f);
        uint32_t ix[P];
#pragma unroll
        for (int p = 0; p < P; ++p) ix[p] = 0;
        Range rg;
        Tail<P> tl;
        tl.bounds = A.seg + (D - 2) * (A.nm1 + 1);
        tl.s = share * A.nseg / A.nshare;
        tl.end = (share + 1) * A.nseg / A.nshare;
        tl.nseg = A.nseg;
        tl.emit = A.emit;
        tl.stride = A.num_evals;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            tl.out[p] = first + 32 * p < end ? A.part_out + first + 32 * p : nullptr;
            tl.valid[p] = valid[p];
            tl.nan_in[p] = nan_in[p];
            tl.part[0][p] = tl.part[1][p] = tl.total[0][p] = tl.total[1][p] = 0.0f;
        }
        rg.lo = tl.s > 0 ? __ldg(tl.bounds + tl.s) : 0u;
        rg.next = tl.s + 1 < A.nseg ? __ldg(tl.bounds + tl.s + 1) : 0xFFFFFFFFu;
        Walk<D, 0, P, SH>::run(G, sx, tid, A.nm1, cur, rg, &tl, in, xC, xA, xB, pin, ix, sum, comp);
        if (A.nseg > 1) {
            while (tl.s < tl.end) {
                (void)close_segment<P>(&tl, sum, comp);
                sum = comp = FV<P>::all(0.0f);
            }
            if (A.emit != SG_EMIT_SUM) return;
            take<P>(tl.total, sum, comp);
        }
    } else {
        uint32_t base[P];
        FV<P> s;
#pragma unroll
        for (int p = 0; p < P; ++p) base[p] = 0;
        block_sum<D, P>(G, A.nm1, in, xC, xA, xB, base, s);
        kahan_add(sum, comp, s);
    }

    const FV<P> res = vsub(sum, comp);
#pragma unroll
    for (int p = 0; p < P; ++p) {
        const int64_t i = first + 32 * p;
        if (i < end) {
            const float r = valid[p] ? res.get(p) : (nan_in[p] ? __int_as_float(0x7fc00000) : 0.0f);
            A.out[A.perm ? A.perm[i] : i] = r;
        }
    }
}

/* Dynamic shared memory of one CTA: the hats of dims A and C (kHatSlots
 * FV<P> per thread), then the prefix coordinates (NPX * P floats per thread). */
template <int D, int P>
constexpr int kSmemBytes = kHatSlots * kThreads * (int)sizeof(FV<P>) + (D >= 4 ? D - 3 : 1) * P * kThreads * 4 +
                           kUpper<D> * 3 * P * kThreads * 4;

template <int D, int P>
__global__ void __launch_bounds__(kThreads, 2) k_evaluate(const EvalArgs A)
{
    extern __shared__ __align__(16) unsigned char smem_ev[];
    FV<P> *shat = reinterpret_cast<FV<P> *>(smem_ev);
    float *sx = reinterpret_cast<float *>(smem_ev + kHatSlots * kThreads * sizeof(FV<P>));
    const int tid = threadIdx.x;
    const int64_t warp = (blockIdx.x * (int64_t)kThreads + tid) >> 5;
    eval_points<D, P, false>(A, A, sx, shat, tid, warp * (32 * P) + (tid & 31), A.num_evals, 0);
}

/* Many grids of the same dimension in one launch: CTA b evaluates the
 * kThreads*P points of grid items[b].x & (2^29-1) starting at point
 * items[b].y.  SH: sums may be shared, bits 29..31 of items[b].x select the
 * share of the segments; without a table of grids the launch is for grid
 * `one`, whose warps are numbered share by share (warps of one share are
 * neighbours: they read the same part of the grid). */
template <int D, int P, bool SH>
__global__ void __launch_bounds__(kThreads, 2)
    k_evaluate_batch(const EvalArgs *__restrict__ grids, const int2 *__restrict__ items, const EvalArgs one)
{
    extern __shared__ __align__(16) unsigned char smem_ev[];
    FV<P> *shat = reinterpret_cast<FV<P> *>(smem_ev);
    float *sx = reinterpret_cast<float *>(smem_ev + kHatSlots * kThreads * sizeof(FV<P>));
    __shared__ EvalArgs sA;
    const int tid = threadIdx.x;
    int share = 0;
    int64_t first, end;
    if (SH && !grids) {
        if (tid == 0) sA = one;
        __syncthreads();
        const int64_t warp = (blockIdx.x * (int64_t)kThreads + tid) >> 5, groups = (sA.num_evals + 32 * P - 1) / (32 * P);
        share = (int)(warp / groups);
        if (share >= sA.nshare) return;
        first = (warp - share * groups) * (32 * P) + (tid & 31);
        end = sA.num_evals;
    } else {
        const int2 item = items[blockIdx.x];
        const uint32_t *src = reinterpret_cast<const uint32_t *>(grids + (item.x & 0x1FFFFFFF));
        uint32_t *dst = reinterpret_cast<uint32_t *>(&sA);
        for (int w = tid; w < (int)(sizeof(EvalArgs) / 4); w += kThreads) dst[w] = src[w];
        __syncthreads();
        if (SH) share = (int)((unsigned)item.x >> 29);
        first = (int64_t)item.y + (tid >> 5) * (32 * P) + (tid & 31);
        end = min((int64_t)item.y + (int64_t)kThreads * P, sA.num_evals);
    }
    const GridView view(sA);
    eval_points<D, P, SH>(sA, view, sx, shat, tid, first, end, share);
}

} // namespace sgeval

/* points per thread: two, the lanes of the packed FP32x2 instructions */
constexpr int kPts = 2;

/* Each launcher also lets its kernel use its dynamic shared memory (above
 * 48 KB for d >= 8) on the current device when called with no work (A or
 * grids NULL, no items): once per device, before the first launch and outside
 * any stream capture. */
#if SG_EVAL_PART == 0
template <int D>
int eval_launch(const EvalArgs *A, void *stream)
{
    using namespace sgeval;
    if (!A)
        return cudaFuncSetAttribute(k_evaluate<D, kPts>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kSmemBytes<D, kPts>);
    const int64_t blocks = (A->num_evals + SG_EVAL_CTA_POINTS - 1) / SG_EVAL_CTA_POINTS;
    if (blocks > 0x7fffffff) return cudaErrorInvalidValue;
    k_evaluate<D, kPts><<<(unsigned)blocks, kThreads, kSmemBytes<D, kPts>, (cudaStream_t)stream>>>(*A);
    sgk_count(1);
    return cudaGetLastError();
}
#elif SG_EVAL_PART == 1
template <int D>
int eval_batch_launch(const EvalArgs *grids, const int2 *items, int nitems, void *stream)
{
    using namespace sgeval;
    if (!grids)
        return cudaFuncSetAttribute(k_evaluate_batch<D, kPts, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kSmemBytes<D, kPts>);
    if (nitems <= 0) return cudaSuccess;
    k_evaluate_batch<D, kPts, false><<<nitems, kThreads, kSmemBytes<D, kPts>, (cudaStream_t)stream>>>(grids, items,
                                                                                                    EvalArgs());
    sgk_count(1);
    return cudaGetLastError();
}
#else
template <int D>
int eval_shared_launch(const EvalArgs *grids, const int2 *items, int nitems, const EvalArgs *one, void *stream)
{
    using namespace sgeval;
    constexpr bool kHas = D >= 4; /* below, every sum is one segment */
    if (!grids && !one)
        return kHas ? cudaFuncSetAttribute(k_evaluate_batch<D, kPts, kHas>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           kSmemBytes<D, kPts>)
                    : cudaSuccess;
    int64_t blocks = nitems;
    if (one) {
        const int64_t warps = (one->num_evals + 32 * kPts - 1) / (32 * kPts) * one->nshare;
        blocks = (warps + kThreads / 32 - 1) / (kThreads / 32);
    }
    if (!kHas || blocks > 0x7fffffff) return cudaErrorInvalidValue;
    if (blocks <= 0) return cudaSuccess;
    k_evaluate_batch<D, kPts, kHas><<<(unsigned)blocks, kThreads, kSmemBytes<D, kPts>, (cudaStream_t)stream>>>(
        one ? nullptr : grids, items, one ? *one : EvalArgs());
    sgk_count(1);
    return cudaGetLastError();
}
#endif

#endif
