/*
 * Batched index bijection on the device: the reference's idx2gp
 * (adaptive_sparse_grid_bench.c:210-243) and gp2idx (c:187-207), one thread
 * per point, with the index tables passed as kernel parameters (constant
 * bank).  Used to sample functions at grid points without a host round trip.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "sg_kernels.h"

namespace {

struct Tables {
    int d, n;
    int lim[SG_MAX_DIMS];
    int64_t dp[SG_MAX_DIMS][SG_MAX_LEVELS];
    int64_t lidx[SG_MAX_LEVELS + 1];
    int64_t plidx[SG_MAX_LEVELS + 1];
};

__global__ void k_idx2gp(const Tables T, const int64_t *__restrict__ index, int *__restrict__ lv_out,
                         int *__restrict__ ix_out, int64_t count)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < count;
         q += (int64_t)gridDim.x * blockDim.x) {
        int64_t idx = index[q];
        int *lv = lv_out + q * T.d, *ix = ix_out + q * T.d;
        if (idx < 0 || idx >= T.lidx[T.n]) {
            for (int k = 0; k < T.d; ++k) lv[k] = ix[k] = -1;
            continue;
        }
        int s = 0;
        while (s < T.n && idx >= T.lidx[s]) ++s;
        --s;
        idx -= T.lidx[s];
        int64_t rest = idx & (((int64_t)1 << s) - 1);
        int64_t pos = idx >> s;
        int lvl[SG_MAX_DIMS];
        int ss = s;
        for (int i = T.d - 1; i >= 1; --i) {
            int level = 0;
            while (pos >= T.dp[i - 1][ss - level]) {
                pos -= T.dp[i - 1][ss - level];
                ++level;
            }
            lvl[i] = level;
            ss -= level;
        }
        lvl[0] = ss;
        for (int i = T.d - 1; i >= 0; --i) {
            lv[i] = lvl[i];
            ix[i] = (int)(rest & (((int64_t)1 << lvl[i]) - 1));
            rest >>= lvl[i];
        }
    }
}

__global__ void k_gp2idx(const Tables T, const int *__restrict__ lv_in, const int *__restrict__ ix_in,
                         int64_t *__restrict__ index, int64_t count)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < count;
         q += (int64_t)gridDim.x * blockDim.x) {
        const int *lv = lv_in + q * T.d, *ix = ix_in + q * T.d;
        int s = 0;
        bool ok = true;
        for (int k = 0; k < T.d; ++k) {
            ok &= lv[k] >= 0 && lv[k] <= T.lim[k] && ix[k] >= 0 && ix[k] < (1 << lv[k]);
            s += lv[k];
        }
        if (!ok || s >= T.n) {
            index[q] = -1;
            continue;
        }
        int64_t in_sub = ix[0], pos = 0;
        int sum = lv[0];
        for (int i = 1; i < T.d; ++i) {
            in_sub = (in_sub << lv[i]) + ix[i];
            sum += lv[i];
            for (int j = 0; j < lv[i]; ++j) pos += T.dp[i - 1][sum - j];
        }
        index[q] = T.lidx[s] + (pos << s) + in_sub;
    }
}

struct FnParams {
    int fn, np;
    double p[SG_MAX_FN_PARAMS];
};

/* f at the grid points, four consecutive elements of the layout per thread.  In
 * a group of level sum s >= 2 they lie in one subspace, so its level vector is
 * found once for the four (it was most of the time, with a double division per
 * coordinate: x_k = (2 i_k + 1) / 2^(l_k+1) is exact, as a product with a power
 * of two too).  d = 6, n = 12 (limits 9, 8), N = 13.3 M, Gaussian bump: see
 * sgk_sample.  Padding between groups is set to 0. */
struct SampleTables {
    int d, n;
    uint32_t dp[SG_MAX_DIMS][SG_MAX_LEVELS];
    uint32_t size[SG_MAX_LEVELS];       /* values of group s         */
    uint32_t start[SG_MAX_LEVELS + 1];  /* first place of group s    */
};

template <int FN>
__device__ __forceinline__ void sample_term(double &acc, double x, int k, const FnParams &F)
{
    if constexpr (FN == SG_FN_REFERENCE) acc += x * x * (1.0 - x) * (1.0 - x);
    else if constexpr (FN == SG_FN_PROD4) acc *= 4.0 * x * (1.0 - x);
    else if constexpr (FN == SG_FN_GAUSS) acc += x * x;
    else if constexpr (FN == SG_FN_BUMP) acc += (x - F.p[0]) * (x - F.p[0]);
    else acc *= F.p[3 * k] + F.p[3 * k + 1] * x + F.p[3 * k + 2] * x * x;
}

/* values q .. q + P - 1 of group s, all in one subspace */
template <int FN, int P>
__device__ __forceinline__ void sample_points(const SampleTables &T, const FnParams &F, int s, uint32_t q, float (&out)[P])
{
    uint32_t pos = q >> s, rest = q & ((1u << s) - 1u);
    double acc[P];
#pragma unroll
    for (int p = 0; p < P; ++p) acc[p] = (FN == SG_FN_PROD4 || FN == SG_FN_QUAD) ? 1.0 : 0.0;
    /* the levels come out last dim first, which is the order of the index
     * bits and of the sums */
    int left = s, shift = 0;
    for (int k = T.d - 1; k >= 0; --k) {
        int l = 0;
        if (k >= 1) {
            uint32_t c = T.dp[k - 1][left];
            while (pos >= c) {
                pos -= c;
                ++l;
                c = T.dp[k - 1][left - l];
            }
        } else {
            l = left;
        }
        left -= l;
        const double scale = __hiloint2double((1022 - l) << 20, 0); /* 2^-(l+1) */
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const uint32_t ik = ((rest + p) >> shift) & ((1u << l) - 1u);
            sample_term<FN>(acc[p], (double)(2 * ik + 1) * scale, k, F);
        }
        shift += l;
    }
#pragma unroll
    for (int p = 0; p < P; ++p) {
        double v = acc[p];
        if (FN == SG_FN_GAUSS) v = exp(-acc[p]);
        if (FN == SG_FN_BUMP) v = exp(-F.p[1] * acc[p]);
        out[p] = __double2float_rn(v);
    }
}

template <int FN>
__global__ void __launch_bounds__(256) k_sample(const SampleTables T, const FnParams F, float *__restrict__ alpha,
                                                int64_t npad)
{
    for (int64_t j = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) * 4; j < npad;
         j += (int64_t)gridDim.x * blockDim.x * 4) {
        int s = T.n - 1;
        while (j < T.start[s]) --s;
        const uint32_t q = (uint32_t)j - T.start[s], size = T.size[s];
        float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (s >= 2) {
            if (q < size) sample_points<FN, 4>(T, F, s, q, v);
        } else {
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                float one[1];
                if (q + p < size) {
                    sample_points<FN, 1>(T, F, s, q + p, one);
                    v[p] = one[0];
                }
            }
        }
        *reinterpret_cast<float4 *>(alpha + j) = make_float4(v[0], v[1], v[2], v[3]);
    }
}

Tables make_tables(const sg_layout *L)
{
    Tables T;
    T.d = L->d;
    T.n = L->n;
    for (int i = 0; i < SG_MAX_DIMS; ++i) T.lim[i] = i < L->d ? L->lim[i] : 0;
    for (int i = 0; i < SG_MAX_DIMS; ++i)
        for (int s = 0; s < SG_MAX_LEVELS; ++s) T.dp[i][s] = L->dp[i][s];
    for (int s = 0; s <= SG_MAX_LEVELS; ++s) T.lidx[s] = L->lidx[s];
    for (int s = 0; s <= SG_MAX_LEVELS; ++s) T.plidx[s] = L->plidx[s];
    return T;
}

} // namespace

extern "C" {

int sgk_idx2gp(const sg_layout *L, const int64_t *index, int *levels, int *indices, int64_t count,
               void *stream)
{
    if (count <= 0) return cudaSuccess;
    int64_t g = (count + 255) / 256;
    if (g > 148 * 16) g = 148 * 16;
    k_idx2gp<<<(unsigned)g, 256, 0, (cudaStream_t)stream>>>(make_tables(L), index, levels, indices,
                                                           count);
    sgk_count(1);
    return cudaGetLastError();
}

int sgk_gp2idx(const sg_layout *L, const int *levels, const int *indices, int64_t *index,
               int64_t count, void *stream)
{
    if (count <= 0) return cudaSuccess;
    int64_t g = (count + 255) / 256;
    if (g > 148 * 16) g = 148 * 16;
    k_gp2idx<<<(unsigned)g, 256, 0, (cudaStream_t)stream>>>(make_tables(L), levels, indices, index,
                                                           count);
    sgk_count(1);
    return cudaGetLastError();
}

int sgk_sample(const sg_layout *L, int fn, const double *params, int nparams, float *alpha, void *stream)
{
    FnParams F;
    F.fn = fn;
    F.np = nparams;
    for (int i = 0; i < SG_MAX_FN_PARAMS; ++i) F.p[i] = i < nparams ? params[i] : 0.0;
    if (L->Npad <= 0) return cudaSuccess;
    SampleTables T;
    T.d = L->d;
    T.n = L->n;
    for (int i = 0; i < SG_MAX_DIMS; ++i)
        for (int q = 0; q < SG_MAX_LEVELS; ++q) T.dp[i][q] = i < L->d && q < L->n ? (uint32_t)L->dp[i][q] : 0;
    for (int q = 0; q <= SG_MAX_LEVELS; ++q) {
        if (q < SG_MAX_LEVELS) T.size[q] = q < L->n ? (uint32_t)(L->lidx[q + 1] - L->lidx[q]) : 0;
        T.start[q] = (uint32_t)L->plidx[q < L->n ? q : L->n];
    }
    int64_t g = (L->Npad / 4 + 255) / 256;
    if (g > 148 * 8) g = 148 * 8;
    cudaStream_t st = (cudaStream_t)stream;
    switch (fn) {
    case SG_FN_REFERENCE: k_sample<SG_FN_REFERENCE><<<(unsigned)g, 256, 0, st>>>(T, F, alpha, L->Npad); break;
    case SG_FN_PROD4: k_sample<SG_FN_PROD4><<<(unsigned)g, 256, 0, st>>>(T, F, alpha, L->Npad); break;
    case SG_FN_GAUSS: k_sample<SG_FN_GAUSS><<<(unsigned)g, 256, 0, st>>>(T, F, alpha, L->Npad); break;
    case SG_FN_BUMP: k_sample<SG_FN_BUMP><<<(unsigned)g, 256, 0, st>>>(T, F, alpha, L->Npad); break;
    case SG_FN_QUAD: k_sample<SG_FN_QUAD><<<(unsigned)g, 256, 0, st>>>(T, F, alpha, L->Npad); break;
    default: return cudaErrorInvalidValue;
    }
    sgk_count(1);
    return cudaGetLastError();
}

} // extern "C"
