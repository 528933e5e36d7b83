/*
 * C ABI of the B200 sparse-grid library (include/sgrid.h).  Host code in C:
 * it owns the handle, the index tables and the device memory, and calls the
 * sm_100a kernels through the launchers of sg_kernels.h.  There is no CPU
 * compute path: every grid operation runs on the GPU, and a missing or
 * unusable GPU is reported as SG_ERR_CUDA.
 */
#include <cuda_runtime_api.h>
#include <pthread.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "sg_kernels.h"
#include "sg_batch_internal.h"
#include "sg_grid_internal.h"
#include "sg_layout.h"

#define SG_API __attribute__((visibility("default")))
#define SG_VERSION "sgb200 0.1.0"

static __thread char g_err[512];

void sg_set_error(const char *fmt, va_list ap) { vsnprintf(g_err, sizeof(g_err), fmt, ap); }

static int fail(int code, const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    sg_set_error(fmt, ap);
    va_end(ap);
    return code;
}

static int cuda_fail(cudaError_t e, const char *what)
{
    return fail(SG_ERR_CUDA, "%s: %s (%s)", what, cudaGetErrorName(e), cudaGetErrorString(e));
}

#define CU(call, what)                                          \
    do {                                                        \
        cudaError_t e_ = (call);                                \
        if (e_ != cudaSuccess) return cuda_fail(e_, what);      \
    } while (0)

SG_API const char *sg_last_error(void) { return g_err; }
SG_API const char *sg_version(void) { return SG_VERSION; }

SG_API int sg_create(int d, int n, const int *limits, sg_grid **grid)
{
    sg_grid *g;
    int r;
    if (!grid) return fail(SG_ERR_ARG, "sg_create: grid is NULL");
    *grid = NULL;
    g = (sg_grid *)calloc(1, sizeof(sg_grid));
    if (!g) return fail(SG_ERR_NOMEM, "sg_create: out of host memory");
    r = sg_layout_init(&g->L, d, n, limits);
    if (r != SG_OK) {
        free(g);
        if (r == SG_ERR_RANGE)
            return fail(r, "sg_create: d=%d n=%d outside 1..%d x 1..%d or grid too large", d, n,
                        SG_MAX_DIMS, SG_MAX_LEVELS);
        return fail(r, "sg_create: invalid arguments d=%d n=%d", d, n);
    }
    g->dev = -1;
    g->opt[SG_OPT_HIER_PRECISION] = SG_HIER_FP32;
    g->opt[SG_OPT_EVAL_SORT] = 1;
    g->opt[SG_OPT_EVAL_PPT] = 0;
    g->opt[SG_OPT_HIER_KERNEL] = 0;
    *grid = g;
    return SG_OK;
}

static void dev_free(sg_grid *g, void *p)
{
    if (!p) return;
    if (g->free_fn) g->free_fn(g->alloc_ctx, p);
    else cudaFree(p);
}

/* ---- memory of shared sums ------------------------------------------------ */

#define SG_SHARE_FLOATS ((int64_t)1 << 25) /* largest buffer of segment sums */
#define SG_POOL_DEVICES 64

/* The segment sums of an evaluation live from its first kernel to its last, on
 * the caller's stream, and evaluations of one handle may overlap on several
 * streams, so each takes its own from a stream-ordered pool: 3 us a call, where
 * growing one buffer took a cudaFree and a cudaMalloc (650 us and a device
 * synchronization), and a smaller call after a larger one does not free what a
 * captured evaluation still names.  One pool per device for all handles; it
 * keeps up to one largest buffer while a handle uses it and gives everything
 * back with the last one.  Streams never wait for one another to reuse memory. */
static pthread_mutex_t g_pool_mu = PTHREAD_MUTEX_INITIALIZER;
static struct {
    cudaMemPool_t pool;
    int users;
} g_pools[SG_POOL_DEVICES];

static void pool_keep(cudaMemPool_t pool, uint64_t bytes)
{
    (void)cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &bytes);
}

static cudaMemPool_t pool_join(int dev)
{
    cudaMemPool_t pool = NULL;
    if (dev >= SG_POOL_DEVICES) return NULL;
    pthread_mutex_lock(&g_pool_mu);
    if (!g_pools[dev].pool) {
        struct cudaMemPoolProps props;
        int off = 0;
        memset(&props, 0, sizeof(props));
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        if (cudaMemPoolCreate(&pool, &props) == cudaSuccess) {
            (void)cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &off);
            g_pools[dev].pool = pool;
        } else {
            cudaGetLastError();
        }
    }
    pool = g_pools[dev].pool;
    if (pool && g_pools[dev].users++ == 0) pool_keep(pool, 4 * SG_SHARE_FLOATS);
    pthread_mutex_unlock(&g_pool_mu);
    return pool;
}

static void pool_leave(int dev)
{
    pthread_mutex_lock(&g_pool_mu);
    if (--g_pools[dev].users == 0) {
        pool_keep(g_pools[dev].pool, 0);
        cudaMemPoolTrimTo(g_pools[dev].pool, 0);
    }
    pthread_mutex_unlock(&g_pool_mu);
}

static void pass_free(sg_grid *g, sg_pass_state *ps)
{
    dev_free(g, ps->units);
    dev_free(g, ps->offs);
    dev_free(g, ps->combos);
    dev_free(g, ps->nodes);
    dev_free(g, ps->combo_of);
    g->dev_bytes -= ps->bytes;
    memset(ps, 0, sizeof(*ps));
}

static void free_device(sg_grid *g)
{
    int k;
    if (g->dev < 0) return;
    cudaSetDevice(g->dev);
    for (k = 0; k < SG_NUM_PHASES; k++)
        if (g->ev[k][0]) {
            cudaEventDestroy(g->ev[k][0]);
            cudaEventDestroy(g->ev[k][1]);
            g->ev[k][0] = g->ev[k][1] = NULL;
        }
    dev_free(g, g->d_alpha);
    dev_free(g, g->d_work);
    dev_free(g, g->d_blk);
    dev_free(g, g->d_repack);
    dev_free(g, g->d_rsrc);
    for (k = 0; k < SG_MAX_DIMS; k++) {
        int f;
        dev_free(g, g->d_chains[k]);
        dev_free(g, g->d_seg[k]);
        for (f = 0; f < 2; f++) pass_free(g, &g->pass[f][k]);
    }
    dev_free(g, g->d_err);
    dev_free(g, g->d_scratch);
    dev_free(g, g->d_io);
    dev_free(g, g->d_sums);
    if (g->sums_pool) pool_leave(g->dev);
    g->sums_pool = NULL;
    while (g->captured) {
        struct sg_captured_sums *c = g->captured;
        g->captured = c->next;
        dev_free(g, c->sums);
        free(c);
    }
}

int sg_create_with_allocator(int d, int n, const int *limits, sg_dev_alloc_fn alloc, sg_dev_free_fn free_fn,
                             void *ctx, sg_grid **grid)
{
    int r;
    if (!alloc || !free_fn) return fail(SG_ERR_ARG, "sg_create_with_allocator: allocator hooks are NULL");
    r = sg_create(d, n, limits, grid);
    if (r != SG_OK) return r;
    (*grid)->alloc = alloc;
    (*grid)->free_fn = free_fn;
    (*grid)->alloc_ctx = ctx;
    return SG_OK;
}

SG_API int sg_destroy(sg_grid *g)
{
    if (!g) return SG_OK;
    free_device(g);
    free(g);
    return SG_OK;
}

SG_API int sg_num_points(const sg_grid *g, int64_t *v)
{
    if (!g || !v) return fail(SG_ERR_ARG, "sg_num_points: NULL argument");
    *v = g->L.N;
    return SG_OK;
}

SG_API int sg_num_subspaces(const sg_grid *g, int64_t *v)
{
    if (!g || !v) return fail(SG_ERR_ARG, "sg_num_subspaces: NULL argument");
    *v = g->L.S;
    return SG_OK;
}

SG_API int sg_dims(const sg_grid *g, int *d, int *n, int *limits)
{
    int k;
    if (!g) return fail(SG_ERR_ARG, "sg_dims: NULL grid");
    if (d) *d = g->L.d;
    if (n) *n = g->L.n;
    if (limits)
        for (k = 0; k < g->L.d; k++) limits[k] = g->L.lim[k];
    return SG_OK;
}

SG_API int sg_tables(const sg_grid *g, int64_t *dp, int64_t *lidx)
{
    int i, s;
    if (!g) return fail(SG_ERR_ARG, "sg_tables: NULL grid");
    if (dp)
        for (i = 0; i < g->L.d; i++)
            for (s = 0; s < g->L.n; s++) dp[i * g->L.n + s] = g->L.dp[i][s];
    if (lidx)
        for (s = 0; s <= g->L.n; s++) lidx[s] = g->L.lidx[s];
    return SG_OK;
}

/* ---- bijection (host) ---------------------------------------------------- */

static int check_levels(const sg_grid *g, const int *lv, int *sum)
{
    int k, s = 0;
    for (k = 0; k < g->L.d; k++) {
        if (lv[k] < 0 || lv[k] > g->L.lim[k]) return 0;
        s += lv[k];
    }
    *sum = s;
    return s <= g->L.n - 1;
}

SG_API int sg_gp2idx(const sg_grid *g, const int *lv, const int *ix, int64_t *index)
{
    int k, s;
    if (!g || !lv || !ix || !index) return fail(SG_ERR_ARG, "sg_gp2idx: NULL argument");
    if (!check_levels(g, lv, &s)) return fail(SG_ERR_ARG, "sg_gp2idx: level vector not in the grid");
    for (k = 0; k < g->L.d; k++)
        if (ix[k] < 0 || ix[k] >= (1 << lv[k])) return fail(SG_ERR_ARG, "sg_gp2idx: index out of range");
    *index = sg_layout_gp2idx(&g->L, lv, ix);
    return SG_OK;
}

SG_API int sg_idx2gp(const sg_grid *g, int64_t index, int *lv, int *ix)
{
    if (!g || !lv || !ix) return fail(SG_ERR_ARG, "sg_idx2gp: NULL argument");
    if (index < 0 || index >= g->L.N) return fail(SG_ERR_ARG, "sg_idx2gp: index %lld out of range", (long long)index);
    return sg_layout_idx2gp(&g->L, index, lv, ix);
}

SG_API int sg_l2idx(const sg_grid *g, const int *lv, int64_t *pos)
{
    int s;
    if (!g || !lv || !pos) return fail(SG_ERR_ARG, "sg_l2idx: NULL argument");
    if (!check_levels(g, lv, &s)) return fail(SG_ERR_ARG, "sg_l2idx: level vector not in the grid");
    *pos = sg_layout_l2idx(&g->L, lv);
    return SG_OK;
}

SG_API int sg_idx2l(const sg_grid *g, int64_t pos, int s, int *lv)
{
    if (!g || !lv) return fail(SG_ERR_ARG, "sg_idx2l: NULL argument");
    if (s < 0 || s >= g->L.n || pos < 0 || pos >= g->L.dp[g->L.d - 1][s])
        return fail(SG_ERR_ARG, "sg_idx2l: position out of range");
    sg_layout_idx2l(&g->L, pos, s, lv);
    return SG_OK;
}

/* ---- device state -------------------------------------------------------- */

static int dev_alloc(sg_grid *g, void **p, int64_t bytes, const char *what)
{
    cudaError_t e;
    if (g->alloc) {
        int r = g->alloc(g->alloc_ctx, p, bytes > 0 ? bytes : 16);
        if (r != SG_OK) {
            *p = NULL;
            return fail(r, "allocating %lld bytes for %s from the handle's allocator", (long long)bytes, what);
        }
        g->dev_bytes += bytes;
        return SG_OK;
    }
    e = cudaMalloc(p, (size_t)(bytes > 0 ? bytes : 16));
    if (e != cudaSuccess) {
        *p = NULL;
        cudaGetLastError();
        return fail(e == cudaErrorMemoryAllocation ? SG_ERR_NOMEM : SG_ERR_CUDA,
                    "cudaMalloc(%lld) for %s: %s", (long long)bytes, what, cudaGetErrorString(e));
    }
    g->dev_bytes += bytes;
    return SG_OK;
}

/* Selects the handle's device for the duration of a call. */
static int enter(sg_grid *g, int *prev)
{
    cudaError_t e = cudaGetDevice(prev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    if (g->dev >= 0 && g->dev != *prev) CU(cudaSetDevice(g->dev), "cudaSetDevice");
    return SG_OK;
}

static void leave(sg_grid *g, int prev)
{
    if (g->dev >= 0 && g->dev != prev) cudaSetDevice(prev);
}

/* A captured evaluation's segment sums: as much for all of a handle's captured
 * calls as for one largest call. */
static void *captured_sums_alloc(sg_grid *g, int64_t floats)
{
    struct sg_captured_sums *c;
    if (g->captured_floats + floats > SG_SHARE_FLOATS) return NULL;
    c = (struct sg_captured_sums *)malloc(sizeof(*c));
    if (!c) return NULL;
    if (dev_alloc(g, &c->sums, floats * 4, "segment sums of a captured evaluation") != SG_OK) {
        free(c);
        return NULL;
    }
    g->captured_floats += floats;
    c->next = g->captured;
    g->captured = c;
    return c->sums;
}

/* Room for one evaluation's segment sums on st, NULL where there is none (whole
 * sums need none).  *ours: to be returned to the pool after the evaluation. */
static float *sums_alloc(sg_grid *g, int64_t floats, cudaStream_t st, int *ours)
{
    enum cudaStreamCaptureStatus cs;
    enum cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    void *p = NULL;
    *ours = 0;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs == cudaStreamCaptureStatusInvalidated) {
        cudaGetLastError();
        return NULL;
    }
    /* st, or another stream of the process, may be capturing: allocating here
     * does not concern it */
    (void)cudaThreadExchangeStreamCaptureMode(&mode);
    if (cs == cudaStreamCaptureStatusActive) {
        p = captured_sums_alloc(g, floats);
    } else {
        if (!g->sums_pool) g->sums_pool = pool_join(g->dev);
        if (g->sums_pool && cudaMallocFromPoolAsync(&p, (size_t)floats * 4, g->sums_pool, st) != cudaSuccess) {
            cudaGetLastError();
            p = NULL;
        }
        *ours = p != NULL;
    }
    (void)cudaThreadExchangeStreamCaptureMode(&mode);
    return (float *)p;
}

/* Undoes a dev_alloc of `bytes` (nothing where *p is NULL). */
static void dev_drop(sg_grid *g, void **p, int64_t bytes)
{
    if (!*p) return;
    dev_free(g, *p);
    g->dev_bytes -= bytes;
    *p = NULL;
}

static int dev_upload(sg_grid *g, void **p, const void *src, int64_t bytes, cudaStream_t st, const char *what)
{
    cudaError_t e;
    int r = dev_alloc(g, p, bytes, what);
    if (r != SG_OK || bytes <= 0) return r;
    /* pageable source: the copy has taken the bytes when the call returns */
    e = cudaMemcpyAsync(*p, src, (size_t)bytes, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) return SG_OK;
    dev_drop(g, p, bytes);
    return cuda_fail(e, what);
}

/* The chain table of dim k (single-dim sweeps). */
static int build_chains(sg_grid *g, int k, cudaStream_t st)
{
    const sg_layout *L = &g->L;
    sg_chain *ch = NULL;
    uint32_t *seg = NULL;
    int64_t nch = 0, nseg = 0, c, cap32 = 0, cap64 = 0;
    int lmax_max = 0, r;
    if (g->d_chains[k]) return SG_OK;
    if ((r = sg_layout_chains(L, k, &ch, &nch, &seg, &nseg)) != SG_OK)
        return fail(r, "building the sweep tables of dim %d", k);
    for (c = 0; c < nch; c++) {
        int j;
        int64_t e32 = 0, e64 = 0;
        for (j = 0; j <= ch[c].lmax; j++) {
            int64_t sz = (int64_t)1 << (ch[c].sigma + j);
            e32 += sz < 4 ? 4 : sz;
            e64 += sz < 2 ? 2 : sz;
        }
        if (e32 > cap32) cap32 = e32;
        if (e64 > cap64) cap64 = e64;
        if (ch[c].lmax > lmax_max) lmax_max = ch[c].lmax;
    }
    r = dev_upload(g, (void **)&g->d_seg[k], seg, nseg * 4, st, "sweep segments");
    if (r == SG_OK)
        r = dev_upload(g, (void **)&g->d_chains[k], ch, nch * (int64_t)sizeof(sg_chain), st, "sweep chains");
    free(ch);
    free(seg);
    if (r != SG_OK) {
        dev_drop(g, (void **)&g->d_seg[k], nseg * 4); /* the next attempt starts afresh */
        return r;
    }
    g->sweep[k].chains = g->d_chains[k];
    g->sweep[k].seg = g->d_seg[k];
    g->sweep[k].nchains = nch;
    g->sweep[k].lmax_max = lmax_max;
    g->sweep[k].cap32 = cap32;
    g->sweep[k].cap64 = cap64;
    return SG_OK;
}

/* The passes of the current precision (f: 0 FP32, 1 FP64): all of them or, on
 * failure, none. */
static int build_passes(sg_grid *g, int f, cudaStream_t st)
{
    const sg_layout *L = &g->L;
    int k, r = SG_OK, n = 0;
    if (g->npass[f]) return SG_OK;
    for (k = 0; k < L->d && r == SG_OK; n++) {
        sg_pass_state *ps = &g->pass[f][n];
        const int64_t before = g->dev_bytes;
        sg_pass_host h;
        const int dims = sg_layout_pass_dims(L, k, f ? 8 : 4);
        ps->k0 = k;
        ps->p.g = dims;
        k += dims ? dims : 1;
        if (!dims) {
            r = build_chains(g, ps->k0, st);
            continue;
        }
        r = sg_layout_pass(L, ps->k0, dims, &h);
        if (r != SG_OK) fail(r, "building the sweep tables of dims %d..%d", ps->k0, k - 1);
        if (r == SG_OK) r = dev_upload(g, (void **)&ps->units, h.units, h.nunits * (int64_t)sizeof(sg_unit), st, "sweep units");
        if (r == SG_OK) r = dev_upload(g, (void **)&ps->offs, h.offs, h.noffs * 4, st, "unit offsets");
        if (r == SG_OK) r = dev_upload(g, (void **)&ps->combos, h.combos, h.ncombos * (int64_t)sizeof(sg_unit_combo), st, "unit levels");
        if (r == SG_OK) r = dev_upload(g, (void **)&ps->nodes, h.nodes, h.nnodes * (int64_t)sizeof(sg_unit_node), st, "unit nodes");
        if (r == SG_OK) r = dev_upload(g, (void **)&ps->combo_of, h.combo_of, h.nall * 2, st, "unit node levels");
        ps->p.units = ps->units;
        ps->p.offs = ps->offs;
        ps->p.nunits = h.nunits;
        ps->p.max_elems = h.max_elems;
        ps->p.tables = h.tables;
        ps->p.tables.combos = ps->combos;
        ps->p.tables.nodes = ps->nodes;
        ps->p.tables.combo_of = ps->combo_of;
        sg_layout_pass_free(&h);
        ps->bytes = g->dev_bytes - before;
    }
    if (r == SG_OK) {
        g->npass[f] = n;
    } else {
        cudaStreamSynchronize(st); /* the uploads of what is freed */
        while (n-- > 0) pass_free(g, &g->pass[f][n]);
    }
    return r;
}

/* The options call for single-dim sweeps throughout. */
static int single_sweeps(const sg_grid *g)
{
    return g->opt[SG_OPT_HIER_KERNEL] == 2 || g->opt[SG_OPT_TEST_WAIT] > 0;
}

/* The sweep tables that the handle's options call for. */
static int sweeps_built(const sg_grid *g)
{
    int k;
    if (!single_sweeps(g)) return g->npass[g->opt[SG_OPT_HIER_PRECISION] == SG_HIER_FP64] > 0;
    for (k = 0; k < g->L.d; k++)
        if (!g->d_chains[k]) return 0;
    return 1;
}

static int build_sweeps(sg_grid *g, cudaStream_t st)
{
    int k, r = SG_OK;
    if (!single_sweeps(g)) return build_passes(g, g->opt[SG_OPT_HIER_PRECISION] == SG_HIER_FP64, st);
    for (k = 0; k < g->L.d && r == SG_OK; k++) r = build_chains(g, k, st);
    return r;
}

/* Allocates the handle's device state and uploads its tables.  The clears
 * and uploads go on `st` (the stream of the call that needs the state, never
 * the legacy default stream, so a serving loop's streams do not wait on
 * them), and the stream is synchronized before returning, so kernels on any
 * stream may read the tables afterwards. */
static int materialize(sg_grid *g, cudaStream_t st)
{
    const sg_layout *L = &g->L;
    sg_repack *rp = NULL;
    uint32_t *rs = NULL, *st_tab = NULL;
    int64_t words;
    int r;
    cudaError_t ce;
    if (g->dev >= 0) return SG_OK;
    CU((cudaError_t)sgk_eval_setup(), "evaluation kernel set-up");
    CU(cudaGetDevice(&g->dev), "cudaGetDevice");
    if ((r = dev_alloc(g, (void **)&g->d_alpha, L->Npad * 4, "grid values")) != SG_OK) goto bad;
    if ((ce = cudaMemsetAsync(g->d_alpha, 0, (size_t)L->Npad * 4, st)) != cudaSuccess) {
        r = cuda_fail(ce, "cudaMemsetAsync");
        goto bad;
    }
    if ((r = dev_alloc(g, (void **)&g->d_err, 16, "error flag")) != SG_OK) goto bad;
    if ((ce = cudaMemsetAsync(g->d_err, 0, 16, st)) != cudaSuccess) {
        r = cuda_fail(ce, "cudaMemsetAsync");
        goto bad;
    }
    if ((r = sg_layout_eval_tables(L, &rp, &rs, g->blk3, g->blk2)) != SG_OK) {
        fail(r, "building the evaluation layout tables");
        goto bad;
    }
    if ((r = dev_alloc(g, (void **)&g->d_blk, L->Nblk * 4, "block layout")) != SG_OK) goto bad;
    if ((r = dev_alloc(g, (void **)&g->d_repack, L->nrows * (int64_t)sizeof(sg_repack), "repack table")) != SG_OK ||
        (r = dev_alloc(g, (void **)&g->d_rsrc, L->S * 4, "repack offsets")) != SG_OK)
        goto bad;
    /* pageable sources: the copies have taken the bytes when the calls return */
    ce = cudaMemcpyAsync(g->d_repack, rp, (size_t)L->nrows * sizeof(sg_repack), cudaMemcpyHostToDevice, st);
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(g->d_rsrc, rs, (size_t)L->S * 4, cudaMemcpyHostToDevice, st);
    if (ce != cudaSuccess) {
        r = cuda_fail(ce, "uploading the repack table");
        goto bad;
    }
    free(rp);
    free(rs);
    rp = NULL;
    rs = NULL;
    if ((words = sg_layout_seg_words(L)) > 0) {
        st_tab = (uint32_t *)malloc((size_t)words * 4);
        if (!st_tab || (r = sg_layout_seg_table(L, g->blk3, st_tab)) != SG_OK) {
            r = fail(SG_ERR_NOMEM, "building the segment table");
            goto bad;
        }
        if ((r = dev_alloc(g, (void **)&g->d_sums, words * 4, "segment table")) != SG_OK) goto bad;
        if ((ce = cudaMemcpyAsync(g->d_sums, st_tab, (size_t)words * 4, cudaMemcpyHostToDevice, st)) != cudaSuccess) {
            r = cuda_fail(ce, "uploading the segment table");
            goto bad;
        }
        free(st_tab);
        st_tab = NULL;
    }
    g->eval_dirty = 1;
    if ((r = build_sweeps(g, st)) != SG_OK) goto bad;
    if ((ce = cudaStreamSynchronize(st)) != cudaSuccess) {
        r = cuda_fail(ce, "uploading the grid tables");
        goto bad;
    }
    return SG_OK;
bad:
    cudaStreamSynchronize(st); /* nothing may still write the ranges freed below */
    free(rp);
    free(rs);
    free(st_tab);
    free_device(g);
    memset(g->d_chains, 0, sizeof(g->d_chains));
    memset(g->d_seg, 0, sizeof(g->d_seg));
    memset(g->pass, 0, sizeof(g->pass));
    memset(g->npass, 0, sizeof(g->npass));
    g->d_alpha = NULL;
    g->d_work = NULL;
    g->d_blk = NULL;
    g->d_repack = NULL;
    g->d_rsrc = NULL;
    g->d_err = NULL;
    g->d_sums = NULL;
    g->d_scratch = g->d_io = NULL;
    g->scratch_bytes = g->io_bytes = g->dev_bytes = 0;
    g->dev = -1;
    return r;
}

/* Whether a kernel on the handle's device may touch the floats [p, p + count):
 * this device's own or managed memory, all inside one allocation, float-aligned.
 * A copy checks or handles the rest (another GPU's memory without peer access,
 * host memory, short buffers, odd addresses); a kernel would fault on it. */
typedef int (*range_fn)(unsigned long long *base, size_t *size, unsigned long long p); /* cuMemGetAddressRange */
static range_fn g_range;
static pthread_once_t g_range_once = PTHREAD_ONCE_INIT;

static void find_range_fn(void)
{
    void *f = NULL;
    enum cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuMemGetAddressRange", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
        g_range = (range_fn)f;
    else
        cudaGetLastError();
}

static int kernel_may_touch(const sg_grid *g, const void *p, int64_t count)
{
    struct cudaPointerAttributes a;
    unsigned long long base = 0, at = (unsigned long long)(uintptr_t)p;
    size_t size = 0;
    if (at % sizeof(float)) return 0;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (a.type != cudaMemoryTypeManaged && !(a.type == cudaMemoryTypeDevice && a.device == g->dev)) return 0;
    pthread_once(&g_range_once, find_range_fn);
    return g_range && g_range(&base, &size, at) == 0 && at + (unsigned long long)count * 4 <= base + size;
}

/* Copies the N compact values into (or out of) the group-aligned layout: one
 * contiguous copy per level group.  Between device buffers one kernel moves the
 * groups below 2^24 values: n copies of two microseconds each were more than
 * half the time of a small grid's hierarchization (d = 4, n = 8: 25 us each way,
 * 4 us in one kernel; d = 10, n = 10: 85 and 65 us).  The copy engine path is
 * the faster one for larger groups (d = 6, n = 14, limits 9: 185 us, 201 us by
 * the kernel), and the one for buffers that the kernel must not touch. */
#define SG_GROUP_COPY ((int64_t)1 << 24)
static int copy_groups(sg_grid *g, float *dst, const float *src, int to_device, enum cudaMemcpyKind kind,
                       cudaStream_t st)
{
    const sg_layout *L = &g->L;
    int s, small = 0, e;
    if (kind == cudaMemcpyDeviceToDevice && kernel_may_touch(g, to_device ? src : dst, L->N)) {
        while (small < L->n && L->lidx[small + 1] - L->lidx[small] < SG_GROUP_COPY) small++;
        if ((e = sgk_copy_groups(L, small, src, dst, !to_device, st)) != cudaSuccess)
            return cuda_fail((cudaError_t)e, "grid values");
    }
    for (s = small; s < L->n; s++) {
        int64_t cnt = L->lidx[s + 1] - L->lidx[s];
        const float *sp;
        float *dp;
        if (cnt == 0) continue;
        sp = to_device ? src + L->lidx[s] : src + L->plidx[s];
        dp = to_device ? dst + L->plidx[s] : dst + L->lidx[s];
        CU(cudaMemcpyAsync(dp, sp, (size_t)cnt * 4, kind, st), "cudaMemcpyAsync (grid values)");
    }
    return SG_OK;
}

SG_API int sg_set_values(sg_grid *g, const float *values)
{
    int prev, r;
    if (!g || !values) return fail(SG_ERR_ARG, "sg_set_values: NULL argument");
    if ((r = enter(g, &prev)) != SG_OK) return r;
    if ((r = materialize(g, 0)) == SG_OK &&
        (r = copy_groups(g, g->d_alpha, values, 1, cudaMemcpyHostToDevice, 0)) == SG_OK) {
        cudaError_t e = cudaStreamSynchronize(0);
        if (e != cudaSuccess) r = cuda_fail(e, "sg_set_values");
        else g->has_values = 1, g->eval_dirty = 1;
    }
    leave(g, prev);
    return r;
}

SG_API int sg_set_values_device(sg_grid *g, const float *values, void *stream)
{
    int prev, r;
    if (!g || !values) return fail(SG_ERR_ARG, "sg_set_values_device: NULL argument");
    if ((r = enter(g, &prev)) != SG_OK) return r;
    if ((r = materialize(g, (cudaStream_t)stream)) == SG_OK &&
        (r = copy_groups(g, g->d_alpha, values, 1, cudaMemcpyDeviceToDevice, (cudaStream_t)stream)) == SG_OK)
        g->has_values = 1, g->eval_dirty = 1;
    leave(g, prev);
    return r;
}

SG_API int sg_get_values(sg_grid *g, float *values)
{
    int prev, r;
    if (!g || !values) return fail(SG_ERR_ARG, "sg_get_values: NULL argument");
    if (!g->has_values) return fail(SG_ERR_STATE, "sg_get_values: no values have been set");
    if ((r = enter(g, &prev)) != SG_OK) return r;
    if ((r = copy_groups(g, values, g->d_alpha, 0, cudaMemcpyDeviceToHost, 0)) == SG_OK)
        r = sg_sync(g, 0);
    leave(g, prev);
    return r;
}

SG_API int sg_get_values_device(sg_grid *g, float *values, void *stream)
{
    int prev, r;
    if (!g || !values) return fail(SG_ERR_ARG, "sg_get_values_device: NULL argument");
    if (!g->has_values) return fail(SG_ERR_STATE, "sg_get_values_device: no values have been set");
    if ((r = enter(g, &prev)) != SG_OK) return r;
    r = copy_groups(g, values, g->d_alpha, 0, cudaMemcpyDeviceToDevice, (cudaStream_t)stream);
    leave(g, prev);
    return r;
}

static void mark(sg_grid *g, int phase, int end, cudaStream_t st)
{
    if (!g->opt[SG_OPT_PROFILE]) return;
    if (!g->ev[phase][0]) {
        if (cudaEventCreate(&g->ev[phase][0]) != cudaSuccess ||
            cudaEventCreate(&g->ev[phase][1]) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
    }
    cudaEventRecord(g->ev[phase][end], st);
    if (end) g->ev_used[phase] = 1;
}

SG_API int sg_timings(sg_grid *g, double *ms)
{
    int k, prev, r;
    if (!g || !ms) return fail(SG_ERR_ARG, "sg_timings: NULL argument");
    for (k = 0; k < SG_NUM_PHASES; k++) ms[k] = -1.0;
    if (g->dev < 0) return SG_OK;
    if ((r = enter(g, &prev)) != SG_OK) return r;
    for (k = 0; k < SG_NUM_PHASES; k++) {
        float t = 0.0f;
        if (!g->ev_used[k]) continue;
        if (cudaEventSynchronize(g->ev[k][1]) != cudaSuccess ||
            cudaEventElapsedTime(&t, g->ev[k][0], g->ev[k][1]) != cudaSuccess) {
            r = cuda_fail(cudaGetLastError(), "sg_timings");
            break;
        }
        ms[k] = t;
    }
    leave(g, prev);
    return r;
}

/* All sweeps of the stored values in place: passes of several dims, and
 * single-dim sweeps where a pass does not apply or the options ask for them. */
static int sweeps_on(sg_grid *g, int f64, cudaStream_t st)
{
    const int kern = (int)g->opt[SG_OPT_HIER_KERNEL], stall = (int)g->opt[SG_OPT_TEST_WAIT];
    int i, k, e;
    if (kern != 2 && stall <= 0) {
        for (i = 0; i < g->npass[f64]; i++) {
            const sg_pass_state *ps = &g->pass[f64][i];
            if (ps->p.g)
                e = f64 ? sgk_sweep_fused_f64(g->d_work, &ps->p, st) : sgk_sweep_fused_f32(g->d_alpha, &ps->p, st);
            else if (sgk_chain_smem_bytes(f64 ? g->sweep[ps->k0].cap64 : g->sweep[ps->k0].cap32, f64 ? 8 : 4) >= 0)
                e = f64 ? sgk_sweep_chains_f64(g->d_work, &g->sweep[ps->k0], g->d_err, st)
                        : sgk_sweep_chains_f32(g->d_alpha, &g->sweep[ps->k0], g->d_err, st);
            else
                e = f64 ? sgk_sweep_gather_f64(g->d_work, &g->sweep[ps->k0], st)
                        : sgk_sweep_gather_f32(g->d_alpha, &g->sweep[ps->k0], st);
            if (e != cudaSuccess) return cuda_fail((cudaError_t)e, "sweep");
        }
        return SG_OK;
    }
    for (k = 0; k < g->L.d; k++) {
        const int fits = sgk_chain_smem_bytes(f64 ? g->sweep[k].cap64 : g->sweep[k].cap32, f64 ? 8 : 4) >= 0;
        if (!f64 && stall > 0 && fits)
            e = sgk_sweep_chains_stall_f32(g->d_alpha, &g->sweep[k], g->d_err, (int64_t)stall << 20, st);
        else if (kern != 2 && fits)
            e = f64 ? sgk_sweep_chains_f64(g->d_work, &g->sweep[k], g->d_err, st)
                    : sgk_sweep_chains_f32(g->d_alpha, &g->sweep[k], g->d_err, st);
        else
            e = f64 ? sgk_sweep_gather_f64(g->d_work, &g->sweep[k], st)
                    : sgk_sweep_gather_f32(g->d_alpha, &g->sweep[k], st);
        if (e != cudaSuccess) return cuda_fail((cudaError_t)e, "sweep");
    }
    return SG_OK;
}

static int hierarchize_on(sg_grid *g, cudaStream_t st)
{
    const sg_layout *L = &g->L;
    int e, r = build_sweeps(g, st); /* built with the values, unless the options changed since */
    if (r != SG_OK) return r;
    if (g->opt[SG_OPT_HIER_PRECISION] != SG_HIER_FP64) return sweeps_on(g, 0, st);
    if (!g->d_work && (r = dev_alloc(g, (void **)&g->d_work, L->Npad * 8, "FP64 working grid")) != SG_OK) return r;
    if ((e = sgk_widen(g->d_alpha, g->d_work, L->Npad, st)) != cudaSuccess) return cuda_fail((cudaError_t)e, "widen");
    if ((r = sweeps_on(g, 1, st)) != SG_OK) return r;
    if ((e = sgk_narrow(g->d_work, g->d_alpha, L->Npad, st)) != cudaSuccess) return cuda_fail((cudaError_t)e, "narrow");
    return SG_OK;
}

SG_API int sg_hierarchize_async(sg_grid *g, void *stream)
{
    int prev, r;
    if (!g) return fail(SG_ERR_ARG, "sg_hierarchize_async: NULL grid");
    if (!g->has_values) return fail(SG_ERR_STATE, "sg_hierarchize: no values have been set");
    if ((r = enter(g, &prev)) != SG_OK) return r;
    mark(g, SG_PHASE_HIERARCHIZE, 0, (cudaStream_t)stream);
    r = hierarchize_on(g, (cudaStream_t)stream);
    g->eval_dirty = 1;
    mark(g, SG_PHASE_HIERARCHIZE, 1, (cudaStream_t)stream);
    leave(g, prev);
    return r;
}

SG_API int sg_hierarchize(sg_grid *g)
{
    int r = sg_hierarchize_async(g, 0);
    if (r != SG_OK) return r;
    return sg_sync(g, 0);
}

/* Device milliseconds of the fastest of `reps` runs of fn on st. */
static int time_best(int (*fn)(sg_grid *, void *), sg_grid *g, void *arg, cudaStream_t st, int reps, double *ms)
{
    cudaEvent_t e0 = NULL, e1 = NULL;
    float t;
    int i, r = SG_OK;
    cudaError_t e = cudaEventCreate(&e0);
    if (e == cudaSuccess) e = cudaEventCreate(&e1);
    *ms = 1e30;
    for (i = 0; e == cudaSuccess && r == SG_OK && i < reps; i++) {
        e = cudaEventRecord(e0, st);
        if (e == cudaSuccess) r = fn(g, arg);
        if (e == cudaSuccess && r == SG_OK) e = cudaEventRecord(e1, st);
        if (e == cudaSuccess && r == SG_OK) e = cudaEventSynchronize(e1);
        if (e == cudaSuccess && r == SG_OK) e = cudaEventElapsedTime(&t, e0, e1);
        if (e == cudaSuccess && r == SG_OK && t < *ms) *ms = t;
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (r == SG_OK && e != cudaSuccess) r = cuda_fail(e, "sg_autotune timing");
    return r;
}

typedef struct tune_eval_arg {
    const float *coords;
    float *out;
    int64_t m;
    cudaStream_t st;
    const float *saved; /* hierarchization: nodal values to restore first */
} tune_eval_arg;

static int tune_eval_once(sg_grid *g, void *a)
{
    const tune_eval_arg *t = (const tune_eval_arg *)a;
    return sg_evaluate_device(g, t->coords, t->out, t->m, t->st);
}

static int tune_hier_once(sg_grid *g, void *a)
{
    const tune_eval_arg *t = (const tune_eval_arg *)a;
    cudaError_t e = cudaMemcpyAsync(g->d_alpha, t->saved, (size_t)g->L.Npad * 4, cudaMemcpyDeviceToDevice, t->st);
    if (e != cudaSuccess) return cuda_fail(e, "sg_autotune restore");
    return hierarchize_on(g, t->st);
}

static int plan_sort(const sg_grid *g, int64_t m);

SG_API int sg_autotune(sg_grid *g, const float *coords, float *out, int64_t num_evals, void *stream, double *ms)
{
    static const int ppts[2] = {1, 2};
    tune_eval_arg ta;
    double t[SG_TUNE_TIMINGS], best = 1e30;
    float *saved = NULL;
    int64_t opt[NOPT];
    int prev, r = SG_OK, i, j, k, chains_apply = 0, bi = -1;
    if (!g || !coords || !out || num_evals < 1) return fail(SG_ERR_ARG, "sg_autotune: bad argument");
    if (!g->has_values) return fail(SG_ERR_STATE, "sg_autotune: no values have been set");
    if ((r = enter(g, &prev)) != SG_OK) return r;
    memcpy(opt, g->opt, sizeof(opt));
    for (i = 0; i < SG_TUNE_TIMINGS; i++) t[i] = -1.0;
    ta.coords = coords;
    ta.out = out;
    ta.m = num_evals;
    ta.st = (cudaStream_t)stream;
    /* evaluation: points per thread x spatial ordering (the per-point
     * arithmetic is the same in every setting, so results do not change) */
    for (i = 0; i < 2 && r == SG_OK; i++)
        for (j = 0; j < 2 && r == SG_OK; j++) {
            g->opt[SG_OPT_EVAL_PPT] = ppts[i];
            g->opt[SG_OPT_EVAL_SORT] = j;
            r = tune_eval_once(g, &ta); /* warm: grows the scratch, builds the block layout */
            if (r == SG_OK) r = time_best(tune_eval_once, g, &ta, ta.st, 2, &t[2 * i + j]);
            if (r == SG_OK && t[2 * i + j] < best) best = t[2 * i + j], bi = 2 * i + j;
        }
    if (r == SG_OK) {
        g->opt[SG_OPT_EVAL_PPT] = ppts[bi / 2];
        /* ordering that is not done at this size was not timed either */
        g->opt[SG_OPT_EVAL_SORT] = 1;
        g->opt[SG_OPT_EVAL_SORT] = plan_sort(g, num_evals) ? bi % 2 : opt[SG_OPT_EVAL_SORT];
    }
    /* under each blocking value (one kernel form: two timings of the same) */
    for (i = 0, best = 1e30, bi = -1; i < SG_EVAL_BLOCKINGS && r == SG_OK; i++) {
        g->opt[SG_OPT_EVAL_BLOCKING] = i + 1;
        r = time_best(tune_eval_once, g, &ta, ta.st, 2, &t[6 + i]);
        if (r == SG_OK && t[6 + i] < best) best = t[6 + i], bi = i;
    }
    if (r == SG_OK) g->opt[SG_OPT_EVAL_BLOCKING] = bi + 1;
    /* hierarchization: shared-memory chains (where they fit) vs gather; the
     * values are saved first and restored at the end */
    if (r == SG_OK) {
        const int f = g->opt[SG_OPT_HIER_PRECISION] == SG_HIER_FP64;
        g->opt[SG_OPT_HIER_KERNEL] = 1;
        r = build_sweeps(g, ta.st);
        for (k = 0; r == SG_OK && k < g->npass[f]; k++) {
            const sg_pass_state *ps = &g->pass[f][k];
            if (ps->p.g || sgk_chain_smem_bytes(f ? g->sweep[ps->k0].cap64 : g->sweep[ps->k0].cap32, f ? 8 : 4) >= 0)
                chains_apply = 1;
        }
    }
    if (r == SG_OK) r = dev_alloc(g, (void **)&saved, g->L.Npad * 4, "sg_autotune saved values");
    if (r == SG_OK) {
        cudaError_t e = cudaMemcpyAsync(saved, g->d_alpha, (size_t)g->L.Npad * 4, cudaMemcpyDeviceToDevice, ta.st);
        if (e != cudaSuccess) r = cuda_fail(e, "sg_autotune save");
        ta.saved = saved;
        for (k = chains_apply ? 1 : 2; k <= 2 && r == SG_OK; k++) {
            g->opt[SG_OPT_HIER_KERNEL] = k;
            r = tune_hier_once(g, &ta);
            if (r == SG_OK) r = time_best(tune_hier_once, g, &ta, ta.st, 2, &t[3 + k]);
        }
        if (r == SG_OK) g->opt[SG_OPT_HIER_KERNEL] = (t[4] >= 0.0 && t[4] <= t[5]) ? 1 : 2;
        e = cudaMemcpyAsync(g->d_alpha, saved, (size_t)g->L.Npad * 4, cudaMemcpyDeviceToDevice, ta.st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ta.st);
        if (r == SG_OK && e != cudaSuccess) r = cuda_fail(e, "sg_autotune restore");
        g->eval_dirty = 1;
    }
    if (saved) dev_free(g, saved);
    if (saved) g->dev_bytes -= g->L.Npad * 4;
    if (r != SG_OK) memcpy(g->opt, opt, sizeof(opt)); /* settings whose tables exist */
    if (ms)
        for (i = 0; i < SG_TUNE_TIMINGS; i++) ms[i] = t[i];
    leave(g, prev);
    return r == SG_OK ? sg_sync(g, stream) : r;
}

SG_API int sg_sync(sg_grid *g, void *stream)
{
    int prev, r = SG_OK, flag = 0;
    cudaError_t e;
    if (!g) return fail(SG_ERR_ARG, "sg_sync: NULL grid");
    if (g->dev < 0) return SG_OK;
    if ((r = enter(g, &prev)) != SG_OK) return r;
    e = cudaMemcpyAsync(&flag, g->d_err, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess) r = cuda_fail(e, "sg_sync");
    else if (flag) {
        cudaMemsetAsync(g->d_err, 0, sizeof(int), (cudaStream_t)stream);
        cudaStreamSynchronize((cudaStream_t)stream);
        r = fail(SG_ERR_TIMEOUT, "a device-side wait gave up; the grid values are not valid");
    }
    leave(g, prev);
    return r;
}

static int ensure(sg_grid *g, void **buf, int64_t *have, int64_t need, const char *what)
{
    int r;
    if (*have >= need) return SG_OK;
    if (*buf) {
        dev_free(g, *buf);
        g->dev_bytes -= *have;
        *buf = NULL;
        *have = 0;
    }
    need = (need + 0xFFFFF) & ~(int64_t)0xFFFFF;
    if ((r = dev_alloc(g, buf, need, what)) != SG_OK) return r;
    *have = need;
    return SG_OK;
}

/* The evaluation plan of the grid's block layout, whole sums. */
static void grid_plan(const sg_grid *g, sg_eval_plan *p)
{
    int k;
    p->alpha = g->d_blk;
    p->d = g->L.d;
    p->n = g->L.n;
    for (k = 0; k < SG_MAX_DIMS; k++) p->lim[k] = k < g->L.d ? g->L.lim[k] : 0;
    for (k = 0; k < SG_MAX_LEVELS; k++) {
        p->blk3[k] = g->blk3[k];
        p->blk2[k] = g->blk2[k];
    }
    p->nseg = g->d_sums ? sg_layout_segs(&g->L) : 1;
    p->nparts = g->d_sums ? sg_layout_parts(&g->L) : 1;
    p->seg = g->d_sums;
    p->nshare = 1;
    p->emit = SG_EMIT_SUM;
    p->part_out = NULL;
}

#define SG_SHARE_ROUNDS 3                  /* resident warps' worth of warps to aim for      */
#define SG_SHARE_MIN_SEGS 4                /* fewer segments: adding them up costs more     */
#define SG_SORT_ROWS ((int64_t)3 << 24)    /* points x rows from which ordering pays        */
#define SG_SORT_BYTES (192 * 1024)         /* block layouts up to an L1 need no ordering    */

/* How many warps share a point's sum.  A launch with few points leaves most of
 * the GPU idle while each thread works through all S subspaces, so where the
 * whole-sum launch would fill less than 3/4 of its rounds of resident warps (16
 * per SM, 64 points each) the segments of a sum go to several warps.  (The
 * kernel that can share is about a quarter slower per point than the one that
 * cannot; above 12 dims, where its walk down to each segment is long, twice as
 * slow, so there only below a quarter: d = 16, n = 5, 65,536 points 1.2 ms whole
 * and 2.1 ms shared before the small subtrees were unrolled there, 0.89 ms whole
 * since.)  d = 10, n = 10: 7.35 -> 0.17 ms for 1,000 points, 6.05 -> 3.3 ms for
 * 65,536; 2^20 points share at a loss (35.3 -> 42.9 ms).  Returns the floats of
 * part_out (0: whole sums).  No choice changes a result. */
static int64_t plan_shares(const sg_grid *g, int64_t m, sg_eval_plan *p)
{
    const int64_t room = (int64_t)sgk_num_sms() * 16, groups = (m + 63) / 64;
    int64_t want, floats;
    /* a pool's grids take no scratch beyond the sort's */
    if (p->nseg < SG_SHARE_MIN_SEGS || g->alloc) return 0;
    if (4 * groups >= (p->d <= 12 ? 3 : 1) * ((groups + room - 1) / room * room)) return 0;
    want = (SG_SHARE_ROUNDS * room + groups - 1) / groups;
    if (want <= p->nparts) {
        p->nshare = p->nparts;
        p->emit = SG_EMIT_PARTS;
        floats = 2 * p->nparts * m;
    } else {
        p->nshare = want < p->nseg ? (int)want : p->nseg;
        p->emit = SG_EMIT_SEGS;
        floats = 2 * p->nseg * m;
    }
    if (floats <= SG_SHARE_FLOATS) return floats;
    p->nshare = 1;
    p->emit = SG_EMIT_SUM;
    return 0;
}

/* Whether to put the points in spatial order first: it makes a warp's gathers
 * share cache lines, at four or more launches.  Measured to pay from about
 * 50 M points x rows on (d = 10, n = 10: 1,000 points; d = 6, n = 8: 65,536), and
 * not at all for a layout that fits L1 (d = 4, n = 8: 2^20 points 136 us in
 * caller order, 171 us ordered).  No choice changes a result. */
static int plan_sort(const sg_grid *g, int64_t m)
{
    return g->opt[SG_OPT_EVAL_SORT] && m * g->L.nrows >= SG_SORT_ROWS && g->L.Nblk * 4 > SG_SORT_BYTES;
}

/* The ordering's scratch regions. */
typedef struct sort_scratch {
    int64_t sort_b, coords_b, perm_b; /* bytes of each */
} sort_scratch;

static int64_t scratch_plan(int64_t m, int d, int sort, sort_scratch *s)
{
    s->sort_b = sort ? (sgk_sort_scratch_bytes(m, d) + 255) & ~(int64_t)255 : 0;
    s->coords_b = sort ? (m * d * 4 + 255) & ~(int64_t)255 : 0;
    s->perm_b = sort ? (m * 4 + 255) & ~(int64_t)255 : 0;
    return s->sort_b + s->coords_b + s->perm_b;
}

static void whole_sums(sg_eval_plan *p)
{
    p->nshare = 1;
    p->emit = SG_EMIT_SUM;
    p->part_out = NULL;
}

/* The evaluation launches; base: the ordering's scratch, where it has any. */
static int evaluate_with(sg_grid *g, sg_eval_plan *p, const sort_scratch *s, char *base, int profile,
                         const float *coords, float *out, int64_t m, cudaStream_t st)
{
    const int32_t *perm = NULL;
    int e;
    if (g->eval_dirty) {
        if ((e = sgk_repack(g->d_alpha, g->d_blk, g->d_repack, g->d_rsrc, g->L.nrows, g->L.n, st)) != cudaSuccess)
            return cuda_fail((cudaError_t)e, "repacking surpluses");
        g->eval_dirty = 0;
    }
    if (s->sort_b) {
        float *sorted = (float *)(base + s->sort_b);
        perm = (const int32_t *)(base + s->sort_b + s->coords_b);
        if (profile) mark(g, SG_PHASE_SORT, 0, st);
        /* the histogram is cleared inside the sort, so nothing left in the
         * scratch by an earlier call is read */
        if ((e = sgk_sort_points(coords, m, p->d, base, sorted, (int32_t *)perm, st)) != cudaSuccess)
            return cuda_fail((cudaError_t)e, "sorting query points");
        if (profile) mark(g, SG_PHASE_SORT, 1, st);
        coords = sorted;
    } else if (profile && g->opt[SG_OPT_PROFILE]) {
        g->ev_used[SG_PHASE_SORT] = 0; /* not a phase of this call */
    }
    if (profile) mark(g, SG_PHASE_EVALUATE, 0, st);
    e = sgk_evaluate(p, coords, perm, out, m, st);
    if (e == cudaSuccess && p->nshare > 1) e = sgk_combine_one(p, perm, out, m, st);
    if (profile) mark(g, SG_PHASE_EVALUATE, 1, st);
    return e == cudaSuccess ? SG_OK : cuda_fail((cudaError_t)e, "evaluate");
}

static int evaluate_on(sg_grid *g, const float *coords, float *out, int64_t m, cudaStream_t st)
{
    sg_eval_plan p;
    sort_scratch s;
    int64_t need, sums;
    int r, ours = 0;
    cudaError_t e;
    grid_plan(g, &p);
    sums = plan_shares(g, m, &p);
    need = scratch_plan(m, p.d, plan_sort(g, m), &s);
    r = need ? ensure(g, &g->d_scratch, &g->scratch_bytes, need, "evaluate scratch") : SG_OK;
    if (r != SG_OK) return r;
    if (sums && !(p.part_out = sums_alloc(g, sums, st, &ours))) whole_sums(&p);
    r = evaluate_with(g, &p, &s, (char *)g->d_scratch, 1, coords, out, m, st);
    if (ours && (e = cudaFreeAsync(p.part_out, st)) != cudaSuccess && r == SG_OK)
        r = cuda_fail(e, "evaluate: returning the segment sums");
    return r;
}

SG_API int sg_evaluate_device(sg_grid *g, const float *coords, float *out, int64_t m, void *stream)
{
    int prev, r;
    if (!g || (m > 0 && (!coords || !out)) || m < 0) return fail(SG_ERR_ARG, "sg_evaluate_device: bad argument");
    if (!g->has_values) return fail(SG_ERR_STATE, "sg_evaluate: no values have been set");
    if (m > 0x7fffffffLL) return fail(SG_ERR_RANGE, "sg_evaluate: at most 2^31-1 points per call");
    if (m == 0) return SG_OK;
    if ((r = enter(g, &prev)) != SG_OK) return r;
    r = evaluate_on(g, coords, out, m, (cudaStream_t)stream);
    leave(g, prev);
    return r;
}

/* The no-allocation evaluation: as evaluate_on with sorting, but every
 * scratch region is carved from the library's fixed device array and no
 * device memory, event or other resource is created. */
SG_API int sg_evaluate_device_noalloc(sg_grid *g, const float *coords, float *out, int64_t m, void *stream)
{
    sg_eval_plan p;
    sort_scratch s;
    int prev, r = SG_OK, e;
    void *scratch = NULL;
    int64_t have = 0, need, sums;
    if (!g || m < 0 || (m > 0 && (!coords || !out))) return fail(SG_ERR_ARG, "sg_evaluate_device_noalloc: bad argument");
    if (!g->has_values || g->dev < 0)
        return fail(SG_ERR_STATE, "sg_evaluate_device_noalloc: the grid has no device state yet (set values first)");
    if (m > SG_NOALLOC_MAX_POINTS)
        return fail(SG_ERR_RANGE, "sg_evaluate_device_noalloc: %lld points exceed SG_NOALLOC_MAX_POINTS (%d)",
                    (long long)m, SG_NOALLOC_MAX_POINTS);
    if (m == 0) return SG_OK;
    if ((r = enter(g, &prev)) != SG_OK) return r;
    grid_plan(g, &p);
    sums = plan_shares(g, m, &p);
    need = scratch_plan(m, g->L.d, plan_sort(g, m), &s);
    if ((e = sgk_noalloc_scratch(&scratch, &have)) != cudaSuccess) {
        r = cuda_fail((cudaError_t)e, "sg_evaluate_device_noalloc: scratch address");
    } else {
        if (sums && need + sums * 4 <= have) p.part_out = (float *)((char *)scratch + need);
        else whole_sums(&p);
        if (need > have)
            r = fail(SG_ERR_RANGE, "sg_evaluate_device_noalloc: %lld points in %d dims need more than the %lld-byte scratch",
                     (long long)m, g->L.d, (long long)have);
        else
            r = evaluate_with(g, &p, &s, (char *)scratch, 0, coords, out, m, (cudaStream_t)stream);
    }
    leave(g, prev);
    return r;
}

SG_API int sg_evaluate(sg_grid *g, const float *coords, float *out, int64_t m)
{
    int prev, r;
    int64_t cb, need;
    float *dc, *dout;
    if (!g || (m > 0 && (!coords || !out)) || m < 0) return fail(SG_ERR_ARG, "sg_evaluate: bad argument");
    if (!g->has_values) return fail(SG_ERR_STATE, "sg_evaluate: no values have been set");
    if (m > 0x7fffffffLL) return fail(SG_ERR_RANGE, "sg_evaluate: at most 2^31-1 points per call");
    if (m == 0) return SG_OK;
    if ((r = enter(g, &prev)) != SG_OK) return r;
    cb = (m * g->L.d * 4 + 255) & ~(int64_t)255;
    need = cb + m * 4;
    if ((r = ensure(g, &g->d_io, &g->io_bytes, need, "evaluate staging")) == SG_OK) {
        dc = (float *)g->d_io;
        dout = (float *)((char *)g->d_io + cb);
        if (cudaMemcpyAsync(dc, coords, (size_t)(m * g->L.d * 4), cudaMemcpyHostToDevice, 0) != cudaSuccess)
            r = cuda_fail(cudaGetLastError(), "sg_evaluate: copying coordinates");
        else if ((r = evaluate_on(g, dc, dout, m, 0)) == SG_OK) {
            if (cudaMemcpyAsync(out, dout, (size_t)(m * 4), cudaMemcpyDeviceToHost, 0) != cudaSuccess)
                r = cuda_fail(cudaGetLastError(), "sg_evaluate: copying results");
            else
                r = sg_sync(g, 0);
        }
    }
    leave(g, prev);
    return r;
}

SG_API int sg_subspace_maxabs(sg_grid *g, float *maxabs)
{
    int prev, r;
    cudaError_t e;
    if (!g || !maxabs) return fail(SG_ERR_ARG, "sg_subspace_maxabs: NULL argument");
    if (!g->has_values) return fail(SG_ERR_STATE, "sg_subspace_maxabs: no values have been set");
    if ((r = enter(g, &prev)) != SG_OK) return r;
    r = ensure(g, &g->d_scratch, &g->scratch_bytes, g->L.S * 4, "subspace statistics");
    if (r == SG_OK) {
        e = (cudaError_t)sgk_subspace_maxabs(&g->L, g->d_alpha, (unsigned *)g->d_scratch, 0);
        if (e == cudaSuccess) e = cudaMemcpyAsync(maxabs, g->d_scratch, (size_t)g->L.S * 4, cudaMemcpyDeviceToHost, 0);
        if (e == cudaSuccess) e = cudaStreamSynchronize(0);
        if (e != cudaSuccess) r = cuda_fail(e, "sg_subspace_maxabs");
    }
    leave(g, prev);
    return r;
}

SG_API int sg_sample_function(sg_grid *g, int fn, const double *params, int np, void *stream)
{
    int prev, r, e, need = 0;
    if (!g || np < 0 || np > SG_MAX_FN_PARAMS || (np > 0 && !params))
        return fail(SG_ERR_ARG, "sg_sample_function: bad argument");
    switch (fn) {
    case SG_FN_REFERENCE: case SG_FN_PROD4: case SG_FN_GAUSS: need = 0; break;
    case SG_FN_BUMP: need = 2; break;
    case SG_FN_QUAD: need = 3 * g->L.d; break;
    default: return fail(SG_ERR_ARG, "sg_sample_function: unknown function %d", fn);
    }
    if (np < need) return fail(SG_ERR_ARG, "sg_sample_function: function %d needs %d parameters", fn, need);
    if ((r = enter(g, &prev)) != SG_OK) return r;
    if ((r = materialize(g, (cudaStream_t)stream)) == SG_OK) {
        if ((e = sgk_sample(&g->L, fn, params, np, g->d_alpha, stream)) != cudaSuccess)
            r = cuda_fail((cudaError_t)e, "sg_sample_function");
        else
            g->has_values = 1, g->eval_dirty = 1;
    }
    leave(g, prev);
    return r;
}

SG_API int sg_idx2gp_device(const sg_grid *g, const int64_t *index, int *levels, int *indices, int64_t count,
                            void *stream)
{
    int e;
    if (!g || count < 0 || (count > 0 && (!index || !levels || !indices)))
        return fail(SG_ERR_ARG, "sg_idx2gp_device: bad argument");
    if ((e = sgk_idx2gp(&g->L, index, levels, indices, count, stream)) != cudaSuccess)
        return cuda_fail((cudaError_t)e, "sg_idx2gp_device");
    return SG_OK;
}

SG_API int sg_gp2idx_device(const sg_grid *g, const int *levels, const int *indices, int64_t *index, int64_t count,
                            void *stream)
{
    int e;
    if (!g || count < 0 || (count > 0 && (!index || !levels || !indices)))
        return fail(SG_ERR_ARG, "sg_gp2idx_device: bad argument");
    if ((e = sgk_gp2idx(&g->L, levels, indices, index, count, stream)) != cudaSuccess)
        return cuda_fail((cudaError_t)e, "sg_gp2idx_device");
    return SG_OK;
}

/* Sets an option that chooses the sweep tables and builds those a live handle
 * lacks, here rather than in a hierarchization that may be under stream
 * capture: on a stream of their own, so that neither the legacy stream's work
 * nor a capture is waited for or disturbed.  On failure the option keeps its
 * value, whose tables exist. */
static int set_sweep_option(sg_grid *g, int option, int64_t value)
{
    const int64_t old = g->opt[option];
    enum cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaStream_t st = NULL;
    cudaError_t e;
    int prev, r = SG_OK;
    g->opt[option] = value;
    if (g->dev < 0 || sweeps_built(g)) return SG_OK;
    if ((r = enter(g, &prev)) == SG_OK) {
        (void)cudaThreadExchangeStreamCaptureMode(&mode);
        if ((e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking)) != cudaSuccess) {
            r = cuda_fail(e, "sg_set_option: stream");
        } else {
            r = build_sweeps(g, st);
            e = cudaStreamSynchronize(st);
            if (r == SG_OK && e != cudaSuccess) r = cuda_fail(e, "uploading sweep tables");
            cudaStreamDestroy(st);
        }
        (void)cudaThreadExchangeStreamCaptureMode(&mode);
        leave(g, prev);
    }
    if (r != SG_OK) g->opt[option] = old;
    return r;
}

SG_API int sg_set_option(sg_grid *g, int option, int64_t value)
{
    if (!g) return fail(SG_ERR_ARG, "sg_set_option: NULL grid");
    switch (option) {
    case SG_OPT_HIER_PRECISION:
        if (value != SG_HIER_FP32 && value != SG_HIER_FP64) return fail(SG_ERR_ARG, "bad precision %lld", (long long)value);
        break;
    case SG_OPT_EVAL_SORT:
        if (value != 0 && value != 1) return fail(SG_ERR_ARG, "SG_OPT_EVAL_SORT is 0 or 1");
        break;
    case SG_OPT_EVAL_PPT:
        if (value < 0 || value > 2) return fail(SG_ERR_ARG, "SG_OPT_EVAL_PPT is 0, 1 or 2");
        break;
    case SG_OPT_HIER_KERNEL:
        if (value < 0 || value > 2) return fail(SG_ERR_ARG, "SG_OPT_HIER_KERNEL is 0, 1 or 2");
        break;
    case SG_OPT_PROFILE:
        if (value != 0 && value != 1) return fail(SG_ERR_ARG, "SG_OPT_PROFILE is 0 or 1");
        break;
    case SG_OPT_TEST_WAIT:
        if (value < 0 || value > 2048) return fail(SG_ERR_ARG, "SG_OPT_TEST_WAIT is 0 .. 2048");
        break;
    case SG_OPT_EVAL_BLOCKING:
        if (value < 0 || value > SG_EVAL_BLOCKINGS) return fail(SG_ERR_ARG, "SG_OPT_EVAL_BLOCKING is 0 .. %d", SG_EVAL_BLOCKINGS);
        break;
    default:
        return fail(SG_ERR_ARG, "unknown option %d", option);
    }
    if (option == SG_OPT_HIER_PRECISION || option == SG_OPT_HIER_KERNEL || option == SG_OPT_TEST_WAIT)
        return set_sweep_option(g, option, value);
    g->opt[option] = value;
    return SG_OK;
}

SG_API int sg_get_option(const sg_grid *g, int option, int64_t *value)
{
    if (!g || !value || option < 1 || option >= NOPT) return fail(SG_ERR_ARG, "sg_get_option: bad argument");
    *value = g->opt[option];
    return SG_OK;
}

SG_API int sg_kernel_launches(int64_t *count)
{
    if (!count) return fail(SG_ERR_ARG, "sg_kernel_launches: NULL argument");
    *count = sgk_launches();
    return SG_OK;
}

SG_API int sg_device_bytes(const sg_grid *g, int64_t *bytes)
{
    if (!g || !bytes) return fail(SG_ERR_ARG, "sg_device_bytes: NULL argument");
    *bytes = g->dev_bytes;
    return SG_OK;
}

/* ---- internal, for the serving loop ------------------------------------- */

int sg_grid_prepare_eval(sg_grid *g, cudaStream_t st)
{
    int e;
    if (!g->eval_dirty) return SG_OK;
    if ((e = sgk_repack(g->d_alpha, g->d_blk, g->d_repack, g->d_rsrc, g->L.nrows, g->L.n, st)) != cudaSuccess)
        return cuda_fail((cudaError_t)e, "repacking surpluses");
    g->eval_dirty = 0;
    return SG_OK;
}

void sg_grid_eval_args(const sg_grid *g, const float *coords, float *out, int64_t m, sg_eval_args *a)
{
    sg_eval_plan p;
    grid_plan(g, &p);
    sgk_fill_eval_args(&p, coords, NULL, out, m, a);
}
