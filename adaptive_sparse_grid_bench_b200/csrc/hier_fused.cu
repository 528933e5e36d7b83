/*
 * Hierarchization sweeps of two or three dims in one pass over the grid.
 *
 * The arithmetic is hierarchize0's (adaptive_sparse_grid_bench.c:557-571): in
 * the sweep of dim k every point with l_k >= 1 becomes a - (left + right) * 0.5
 * from the values before that sweep, dim after dim.  The subspaces that
 * differ only in the levels of the pass's dims form a unit that the pass's
 * sweeps never leave, so one CTA reads a unit, runs all its sweeps in shared
 * memory in dim order, and writes it back: a pass moves the grid once instead
 * of once per dim, and the results are the same bits.
 *
 * A unit is 2^sigma independent cells (index combinations of the other dims),
 * each a small sparse grid of the pass's dims with level budget R.  In shared
 * memory it is stored node by node, a node's cells side by side: a node
 * (levels and indices of the pass's dims) has the same two parents in every
 * cell, so one table entry drives the updates of all its cells and every
 * access is a contiguous row.  A sweep goes from the finest level to the
 * coarsest with a barrier between levels, so a point's parents, all coarser,
 * still hold their values from before it.
 *
 * What bounds it: the grid's traffic through L2 per pass.  d = 10, n = 10 (N =
 * 33.0 M) reads 27 M and writes 25 M values per pass of two dims, five passes,
 * against 20.5 M read and 16.2 M written by each of ten single-dim sweeps
 * whose CTAs spent 350 instructions per warp and chain on set-up.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "sg_kernels.h"

namespace {

__device__ __forceinline__ float upd(float a, float l, float r)
{
    return __fsub_rn(a, __fmul_rn(__fadd_rn(l, r), 0.5f));
}
__device__ __forceinline__ double upd(double a, double l, double r)
{
    return __dsub_rn(a, __dmul_rn(__dadd_rn(l, r), 0.5));
}

/* W elements of T moved at once: 16 bytes, or one */
template <typename T, int W>
struct Vec {
    static_assert(W == 1, "one element");
    using type = T;
    static __device__ __forceinline__ T zero() { return T(0); }
    static __device__ __forceinline__ void scatter(T *r, int, int, T x) { *r = x; }
    static __device__ __forceinline__ T gather(const T *r, int, int) { return *r; }
};
template <>
struct Vec<float, 4> {
    using type = float4;
    static __device__ __forceinline__ float4 zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
    static __device__ __forceinline__ void scatter(float *r, int w1, int w2, float4 x)
    {
        r[0] = x.x;
        r[w1] = x.y;
        r[w2] = x.z;
        r[w1 + w2] = x.w;
    }
    static __device__ __forceinline__ float4 gather(const float *r, int w1, int w2)
    {
        return make_float4(r[0], r[w1], r[w2], r[w1 + w2]);
    }
};
template <>
struct Vec<double, 2> {
    using type = double2;
    static __device__ __forceinline__ double2 zero() { return make_double2(0.0, 0.0); }
    static __device__ __forceinline__ void scatter(double *r, int w1, int, double2 x)
    {
        r[0] = x.x;
        r[w1] = x.y;
    }
    static __device__ __forceinline__ double2 gather(const double *r, int w1, int) { return make_double2(r[0], r[w1]); }
};
__device__ __forceinline__ float4 upd(float4 a, float4 l, float4 r)
{
    return make_float4(upd(a.x, l.x, r.x), upd(a.y, l.y, r.y), upd(a.z, l.z, r.z), upd(a.w, l.w, r.w));
}
__device__ __forceinline__ double2 upd(double2 a, double2 l, double2 r)
{
    return make_double2(upd(a.x, l.x, r.x), upd(a.y, l.y, r.y));
}

/* Where element q of a subspace goes whose levels in the pass's dims sum to L:
 * its cell (the index bits above and below those of the pass's consecutive
 * dims) in the row of its node. */
__device__ __forceinline__ int place(int q, int L, int lo, int stride)
{
    return ((q >> lo) & ((1 << L) - 1)) * stride + ((q & ((1 << lo) - 1)) | ((q >> (lo + L)) << lo));
}

/* Copies the unit between global and shared memory, W elements (16 bytes) per
 * thread and step, kAhead steps' loads in flight.  A node's cells are a
 * contiguous run of 2^sigma values in its subspace when the index bits are
 * counted in memory order, so run n of the unit is found through the combo that
 * node n belongs to; its values scatter to the rows of several nodes.  ROW: the
 * dims after the pass's give the lowest W cells, so the W elements are
 * neighbours in one node's row and move at once (scattered one by one they cost
 * four times the instructions and, four banks apart, sixteen times the
 * shared-memory cycles). */
constexpr int kAhead = 4;
template <typename T, int NT, int W, bool ROW>
__device__ __forceinline__ void load_unit(const T *__restrict__ a, T *buf, const sg_unit &u,
                                          const uint32_t *__restrict__ off, const sg_unit_tables &tb, int nodes,
                                          int stride)
{
    using V = typename Vec<T, W>::type;
    const int sv = u.sigma - (W == 4 ? 2 : W - 1), lo = u.lo, total = nodes << sv;
    for (int v0 = threadIdx.x; v0 < total; v0 += NT * kAhead) {
        V x[kAhead];
        int at[kAhead], w1[kAhead], w2[kAhead];
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
            const int v = v0 + i * NT;
            if (v < total) {
                const int n = v >> sv, c = __ldg(tb.combo_of + n);
                const sg_unit_combo cb = tb.combos[c];
                const int q = ((n - (int)cb.node) << u.sigma) + (v & ((1 << sv) - 1)) * W;
                x[i] = *reinterpret_cast<const V *>(a + __ldg(off + c) + q);
                at[i] = (int)cb.node * stride + place(q, cb.sum, lo, stride);
                w1[i] = W > 1 && !ROW ? place(1, cb.sum, lo, stride) : 0;
                w2[i] = W > 2 && !ROW ? place(2, cb.sum, lo, stride) : 0;
            }
        }
#pragma unroll
        for (int i = 0; i < kAhead; ++i)
            if (v0 + i * NT < total) {
                if (ROW) *reinterpret_cast<V *>(buf + at[i]) = x[i];
                else Vec<T, W>::scatter(buf + at[i], w1[i], w2[i], x[i]);
            }
    }
}

template <typename T, int NT, int W, bool ROW>
__device__ __forceinline__ void store_unit(T *__restrict__ a, const T *buf, const sg_unit &u,
                                           const uint32_t *__restrict__ off, const sg_unit_tables &tb, int nodes,
                                           int stride)
{
    using V = typename Vec<T, W>::type;
    const int sv = u.sigma - (W == 4 ? 2 : W - 1), lo = u.lo, total = nodes << sv;
    /* node 0, the subspace of levels 0, never changes */
    for (int v = (1 << sv) + threadIdx.x; v < total; v += NT) {
        const int n = v >> sv, c = __ldg(tb.combo_of + n);
        const sg_unit_combo cb = tb.combos[c];
        const int q = ((n - (int)cb.node) << u.sigma) + (v & ((1 << sv) - 1)) * W;
        const T *r = buf + ((int)cb.node * stride + place(q, cb.sum, lo, stride));
        *reinterpret_cast<V *>(a + __ldg(off + c) + q) =
            ROW ? *reinterpret_cast<const V *>(r) : Vec<T, W>::gather(r, W > 1 ? place(1, cb.sum, lo, stride) : 0, W > 2 ? place(2, cb.sum, lo, stride) : 0);
    }
}

/* the sweeps of the pass's dims, W cells per step */
template <typename T, int G, int NT, int W>
__device__ __forceinline__ void sweep_unit(T *buf, const sg_unit &u, const sg_unit_tables &tb, int stride)
{
    using V = typename Vec<T, W>::type;
    const int sv = u.sigma - (W == 4 ? 2 : W - 1);
#pragma unroll
    for (int q = 0; q < G; ++q) {
        for (int j = min((int)u.R, tb.lmax[q]); j >= 1; --j) {
            const sg_unit_node *list = tb.nodes + tb.first[q][j];
            const int items = tb.count[q][j][u.R] << sv;
#pragma unroll 2
            for (int it = threadIdx.x; it < items; it += NT) {
                const sg_unit_node e = list[it >> sv];
                T *col = buf + (it & ((1 << sv) - 1)) * W;
                V *self = reinterpret_cast<V *>(col + (int)e.node * stride), l = Vec<T, W>::zero(), r = l;
                if (e.left != SG_UNIT_NONE) l = *reinterpret_cast<const V *>(col + (int)e.left * stride);
                if (e.right != SG_UNIT_NONE) r = *reinterpret_cast<const V *>(col + (int)e.right * stride);
                *self = upd(*self, l, r);
            }
            __syncthreads();
        }
    }
}

template <typename T, int G, int NT>
__global__ void __launch_bounds__(NT) k_sweep_fused(T *__restrict__ a, const sg_unit *__restrict__ units,
                                                   const uint32_t *__restrict__ offs, const sg_unit_tables tb)
{
    constexpr int W = 16 / (int)sizeof(T);
    extern __shared__ __align__(16) unsigned char smem_fused[];
    T *buf = reinterpret_cast<T *>(smem_fused);
    const sg_unit u = units[blockIdx.x];
    const int stride = sgk_unit_stride(u.sigma), nodes = tb.nnode[u.R];
    const uint32_t *off = offs + u.off;
    if (u.lo >= (W == 4 ? 2 : 1)) {
        load_unit<T, NT, W, true>(a, buf, u, off, tb, nodes, stride);
        __syncthreads();
        sweep_unit<T, G, NT, W>(buf, u, tb, stride);
        store_unit<T, NT, W, true>(a, buf, u, off, tb, nodes, stride);
    } else if (u.sigma >= 2) {
        load_unit<T, NT, W, false>(a, buf, u, off, tb, nodes, stride);
        __syncthreads();
        sweep_unit<T, G, NT, W>(buf, u, tb, stride);
        store_unit<T, NT, W, false>(a, buf, u, off, tb, nodes, stride);
    } else {
        load_unit<T, NT, 1, true>(a, buf, u, off, tb, nodes, stride);
        __syncthreads();
        sweep_unit<T, G, NT, 1>(buf, u, tb, stride);
        store_unit<T, NT, 1, true>(a, buf, u, off, tb, nodes, stride);
    }
}

template <typename T, int G, int NT>
int launch_nt(T *a, const sg_unit_pass *p, cudaStream_t st)
{
    const int64_t smem = p->max_elems * (int64_t)sizeof(T);
    /* the limit is one for the process, so always the same value: set to this
     * launch's size it could be lowered by another thread before the launch */
    cudaError_t e = cudaFuncSetAttribute(k_sweep_fused<T, G, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         SG_UNIT_MAX_BYTES);
    if (e != cudaSuccess) return e;
    k_sweep_fused<T, G, NT><<<(unsigned)p->nunits, NT, (size_t)smem, st>>>(a, p->units, p->offs, p->tables);
    sgk_count(1);
    return cudaGetLastError();
}

/* CTA size by the largest unit, which is one CTA's serial work */
template <typename T, int G>
int launch(T *a, const sg_unit_pass *p, cudaStream_t st)
{
    if (p->max_elems <= 1536) return launch_nt<T, G, 128>(a, p, st);
    if (p->max_elems <= 12 * 1024) return launch_nt<T, G, 256>(a, p, st);
    return launch_nt<T, G, 512>(a, p, st);
}

template <typename T>
int launch_any(T *a, const sg_unit_pass *p, void *stream)
{
    if (p->nunits <= 0) return cudaSuccess;
    if (p->max_elems * (int64_t)sizeof(T) > SG_UNIT_MAX_BYTES) return cudaErrorInvalidValue;
    switch (p->g) {
    case 1: return launch<T, 1>(a, p, (cudaStream_t)stream);
    case 2: return launch<T, 2>(a, p, (cudaStream_t)stream);
    case 3: return launch<T, 3>(a, p, (cudaStream_t)stream);
    default: return cudaErrorInvalidValue;
    }
}

} // namespace

extern "C" int sgk_sweep_fused_f32(float *a, const sg_unit_pass *p, void *stream)
{
    return launch_any<float>(a, p, stream);
}
extern "C" int sgk_sweep_fused_f64(double *a, const sg_unit_pass *p, void *stream)
{
    return launch_any<double>(a, p, stream);
}
