// Per-subspace maximum |surplus| on the device: the statistic the
// limits-adaptive refinement driver (sgrid_refine.c) decides on.
//
// In the group-aligned compact layout the subspaces of level group s follow
// each other, 2^s values each, from a multiple of 32.  A warp takes 1024 values
// of a group, 16 bytes per lane and step, all loads first: up to s = 10 it holds
// whole subspaces and writes each one's maximum, above that one atomic per 1024
// values (with one per 32 the atomics were most of the time).  One pass,
// HBM-bound: 4 bytes read per value, 4 written per subspace.
#include <cuda_runtime.h>
#include <stdint.h>

#include "sg_kernels.h"

namespace {

constexpr int kChunk = 1024, kSteps = kChunk / 128;

struct MaxAbsTables {
    int n;
    int64_t plidx[SG_MAX_LEVELS];     // device offset of group s
    int64_t len[SG_MAX_LEVELS];       // values in group s (multiple of 2^s)
    int64_t sbase[SG_MAX_LEVELS];     // subspaces before group s
    int64_t chunk0[SG_MAX_LEVELS + 1]; // chunks before group s
};

__global__ void __launch_bounds__(256) k_subspace_maxabs(MaxAbsTables T, const float *__restrict__ a,
                                                         unsigned *__restrict__ out)
{
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t c = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < T.chunk0[T.n]; c += nw) {
        int s = T.n - 1;
        while (c < T.chunk0[s]) --s;
        const int64_t first = (c - T.chunk0[s]) * kChunk, len = T.len[s];
        const float *src = a + T.plidx[s] + first;
        unsigned *o = out + T.sbase[s];
        float v[kSteps];
        if (s >= 2) {
            // len is a multiple of 4: a lane's four values are all in the group or none
#pragma unroll
            for (int t = 0; t < kSteps; ++t) {
                const int e = t * 128 + lane * 4;
                v[t] = 0.f;
                if (first + e < len) {
                    const float4 x = __ldg(reinterpret_cast<const float4 *>(src + e));
                    v[t] = fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w)));
                }
            }
            if (s >= 6) {
                // A NaN counts where it fills a run of 32 values: the maximum
                // inside a run passes NaN over, the one over runs compares bit
                // patterns, which put NaN above infinity.  Without NaN (one
                // vote per chunk) both are the same maximum.
                bool nan = false;
                unsigned u[kSteps];
#pragma unroll
                for (int t = 0; t < kSteps; ++t) nan |= v[t] != v[t];
                if (__any_sync(0xffffffffu, nan)) {
#pragma unroll
                    for (int t = 0; t < kSteps; ++t)
                        for (int off = 1; off < 8; off <<= 1)
                            v[t] = fmaxf(v[t], __shfl_xor_sync(0xffffffffu, v[t], off));
                }
#pragma unroll
                for (int t = 0; t < kSteps; ++t) u[t] = __float_as_uint(v[t]); // non-negative: ordered like the floats
                if (s == 6) {
#pragma unroll
                    for (int t = 0; t < kSteps; ++t) {
                        unsigned m = u[t];
                        for (int off = 1; off < 16; off <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, off));
                        const int64_t e = first + t * 128 + lane * 4;
                        if (e < len && (lane & 15) == 0) o[e >> 6] = m;
                    }
                    continue;
                }
                // 2^(s-7) steps per subspace
                const int per = s >= 10 ? kSteps : 1 << (s - 7);
                unsigned m = 0;
#pragma unroll
                for (int t = 0; t < kSteps; ++t) {
                    m = max(m, u[t]);
                    if ((t + 1) % per) continue;
                    for (int off = 16; off; off >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, off));
                    const int64_t e = first + (int64_t)(t + 1 - per) * 128;
                    if (lane == 0 && e < len) {
                        if (s > 10) atomicMax(o + (e >> s), m);
                        else o[e >> s] = m;
                    }
                    m = 0;
                }
            } else {
                // 2^(s-2) lanes per subspace
#pragma unroll
                for (int t = 0; t < kSteps; ++t) {
                    float m = v[t];
                    for (int off = 1; off < 1 << (s - 2); off <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
                    const int64_t e = first + t * 128 + lane * 4;
                    if (e < len && (lane & ((1 << (s - 2)) - 1)) == 0) o[e >> s] = __float_as_uint(m);
                }
            }
        } else {
            for (int e = lane << s; e < kChunk; e += 32 << s) {
                if (first + e >= len) break;
                float m = fabsf(__ldg(src + e));
                if (s == 1) m = fmaxf(m, fabsf(__ldg(src + e + 1)));
                o[(first + e) >> s] = __float_as_uint(m);
            }
        }
    }
}

} // namespace

extern "C" int sgk_subspace_maxabs(const sg_layout *L, const float *alpha, unsigned *out, void *stream)
{
    MaxAbsTables T;
    int64_t sb = 0;
    cudaError_t e;
    T.n = L->n;
    T.chunk0[0] = 0;
    for (int s = 0; s < SG_MAX_LEVELS; ++s) {
        T.plidx[s] = s < L->n ? L->plidx[s] : L->Npad;
        T.len[s] = s < L->n ? L->lidx[s + 1] - L->lidx[s] : 0;
        T.sbase[s] = sb;
        sb += T.len[s] >> s;
        T.chunk0[s + 1] = T.chunk0[s] + (T.len[s] + kChunk - 1) / kChunk;
    }
    if (L->S <= 0 || L->Npad <= 0) return cudaSuccess;
    e = cudaMemsetAsync(out, 0, (size_t)L->S * sizeof(unsigned), (cudaStream_t)stream);
    if (e != cudaSuccess) return e;
    int64_t g = (T.chunk0[L->n] + 7) / 8;
    if (g > 148 * 8) g = 148 * 8;
    k_subspace_maxabs<<<(unsigned)g, 256, 0, (cudaStream_t)stream>>>(T, alpha, out);
    sgk_count(1);
    return cudaGetLastError();
}
