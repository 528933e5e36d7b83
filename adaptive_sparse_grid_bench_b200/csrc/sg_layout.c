/*
 * Host-side index algebra (C).  Follows the reference benchmark
 * adaptive_sparse_grid_bench.c: tables c:101-140 (with the limit handling of
 * the CUDA host code, adaptive_sparse_grid_bench_cuda.cu:79-102), bijection
 * c:187-279.  Also builds the per-sweep chain tables and the evaluation
 * order table that the kernels walk.
 */
#include "sg_layout.h"

#include <stdlib.h>
#include <string.h>

static int64_t block_layout_size(const sg_layout *L);

int sg_layout_init(sg_layout *L, int d, int n, const int *limits)
{
    int i, s, k;
    if (!L || d < 1 || n < 1) return SG_ERR_ARG;
    if (d > SG_MAX_DIMS || n > SG_MAX_LEVELS) return SG_ERR_RANGE;
    memset(L, 0, sizeof(*L));
    L->d = d;
    L->n = n;
    for (i = 0; i < d; i++) {
        int v = limits ? limits[i] : n - 1;
        if (v < 0) return SG_ERR_ARG;
        L->lim[i] = v > n - 1 ? n - 1 : v;
    }
    /* dp[i][s] = sum_{k <= min(s, lim_i)} dp[i-1][s-k]  (c:113-129) */
    for (s = 0; s < n; s++) L->dp[0][s] = s <= L->lim[0];
    for (i = 1; i < d; i++)
        for (s = 0; s < n; s++) {
            int64_t c = 0;
            for (k = 0; k <= s && k <= L->lim[i]; k++) c += L->dp[i - 1][s - k];
            L->dp[i][s] = c;
        }
    /* group offsets (c:132-140), compact and padded */
    L->N = L->S = L->Npad = 0;
    for (s = 0; s < n; s++) {
        int64_t sz = L->dp[d - 1][s] << s;
        L->lidx[s] = L->N;
        L->plidx[s] = L->Npad;
        L->N += sz;
        L->S += L->dp[d - 1][s];
        L->Npad += (sz + SG_GROUP_ALIGN - 1) / SG_GROUP_ALIGN * SG_GROUP_ALIGN;
    }
    L->lidx[n] = L->N;
    L->plidx[n] = L->Npad;
    /* kernels index the device grid with 32-bit offsets */
    if (L->Npad >= ((int64_t)1 << 31)) return SG_ERR_RANGE;
    L->Nblk = block_layout_size(L);
    L->nrows = 0;
    for (s = 0; s < n; s++) L->nrows += d >= 2 ? L->dp[d - 2][s] : s == 0;
    if (L->Nblk >= ((int64_t)1 << 32) - 64) return SG_ERR_RANGE;
    return SG_OK;
}

/* c:266-279 */
int64_t sg_layout_l2idx(const sg_layout *L, const int *lv)
{
    int64_t pos = 0;
    int i, j, sum = lv[0];
    for (i = 1; i < L->d; i++) {
        sum += lv[i];
        for (j = 0; j < lv[i]; j++) pos += L->dp[i - 1][sum - j];
    }
    return pos;
}

/* c:245-264 */
void sg_layout_idx2l(const sg_layout *L, int64_t pos, int s, int *lv)
{
    int i;
    for (i = L->d - 1; i >= 1; i--) {
        int level = 0;
        while (pos >= L->dp[i - 1][s - level]) {
            pos -= L->dp[i - 1][s - level];
            level++;
        }
        lv[i] = level;
        s -= level;
    }
    lv[0] = s;
}

/* c:187-207 */
int64_t sg_layout_gp2idx(const sg_layout *L, const int *lv, const int *ix)
{
    int64_t in_sub = ix[0];
    int i, s = lv[0];
    for (i = 1; i < L->d; i++) {
        in_sub = (in_sub << lv[i]) + ix[i];
        s += lv[i];
    }
    return L->lidx[s] + (sg_layout_l2idx(L, lv) << s) + in_sub;
}

/* c:210-243 */
int sg_layout_idx2gp(const sg_layout *L, int64_t idx, int *lv, int *ix)
{
    int s = 0, i;
    int64_t rest;
    if (idx < 0 || idx >= L->N) return SG_ERR_ARG;
    while (s < L->n && idx >= L->lidx[s]) s++;
    s--;
    idx -= L->lidx[s];
    rest = idx & (((int64_t)1 << s) - 1);
    sg_layout_idx2l(L, idx >> s, s, lv);
    for (i = L->d - 1; i >= 0; i--) {
        ix[i] = (int)(rest & (((int64_t)1 << lv[i]) - 1));
        rest >>= lv[i];
    }
    return SG_OK;
}

int64_t sg_layout_subspace_offset(const sg_layout *L, const int *lv)
{
    int i, s = 0;
    for (i = 0; i < L->d; i++) s += lv[i];
    return L->plidx[s] + (sg_layout_l2idx(L, lv) << s);
}

/* Odometer over level vectors of the dims in `dims` (count m) with sum <= cap
 * and per-dim limits; calls back with the vector written into lv. */
typedef void (*lv_visit)(void *ctx, int *lv, int sum);

static void enum_levels(const sg_layout *L, const int *dims, int m, int idx, int cap,
                        int sum, int *lv, lv_visit fn, void *ctx)
{
    int l, k;
    if (idx == m) {
        fn(ctx, lv, sum);
        return;
    }
    k = dims[idx];
    for (l = 0; l <= L->lim[k] && sum + l <= cap; l++) {
        lv[k] = l;
        enum_levels(L, dims, m, idx + 1, cap, sum + l, lv, fn, ctx);
    }
    lv[k] = 0;
}

typedef struct {
    const sg_layout *L;
    int k;
    sg_chain *chains;
    int64_t nch, cap_ch;
    uint32_t *seg;
    int64_t nseg, cap_seg;
    int err;
} chain_ctx;

static void chain_visit(void *vctx, int *lv, int sigma)
{
    chain_ctx *c = (chain_ctx *)vctx;
    const sg_layout *L = c->L;
    int k = c->k, j, m, lo = 0;
    int lmax = L->n - 1 - sigma;
    if (lmax > L->lim[k]) lmax = L->lim[k];
    if (lmax < 1 || c->err) return;
    if (c->nch == c->cap_ch) {
        c->cap_ch = c->cap_ch ? 2 * c->cap_ch : 1024;
        c->chains = (sg_chain *)realloc(c->chains, (size_t)c->cap_ch * sizeof(sg_chain));
        if (!c->chains) { c->err = SG_ERR_NOMEM; return; }
    }
    while (c->nseg + lmax + 1 > c->cap_seg) {
        c->cap_seg = c->cap_seg ? 2 * c->cap_seg : 4096;
        c->seg = (uint32_t *)realloc(c->seg, (size_t)c->cap_seg * sizeof(uint32_t));
        if (!c->seg) { c->err = SG_ERR_NOMEM; return; }
    }
    for (m = k + 1; m < L->d; m++) lo += lv[m];
    c->chains[c->nch].seg = (uint32_t)c->nseg;
    c->chains[c->nch].sigma = (uint8_t)sigma;
    c->chains[c->nch].lmax = (uint8_t)lmax;
    c->chains[c->nch].lo = (uint8_t)lo;
    c->chains[c->nch].pad = 0;
    c->nch++;
    for (j = 0; j <= lmax; j++) {
        lv[k] = j;
        c->seg[c->nseg++] = (uint32_t)sg_layout_subspace_offset(L, lv);
    }
    lv[k] = 0;
}

static int chain_size_cmp(const void *a, const void *b)
{
    const sg_chain *x = (const sg_chain *)a, *y = (const sg_chain *)b;
    /* size = 2^sigma * (2^(lmax+1) - 1); compare exactly */
    int64_t sx = ((int64_t)1 << x->sigma) * (((int64_t)2 << x->lmax) - 1);
    int64_t sy = ((int64_t)1 << y->sigma) * (((int64_t)2 << y->lmax) - 1);
    if (sx != sy) return sx > sy ? -1 : 1;
    return x->seg < y->seg ? -1 : (x->seg > y->seg);
}

int sg_layout_chains(const sg_layout *L, int k, sg_chain **chains, int64_t *nchains,
                     uint32_t **seg_off, int64_t *nseg)
{
    int dims[SG_MAX_DIMS], lv[SG_MAX_DIMS], m = 0, i;
    chain_ctx c;
    memset(&c, 0, sizeof(c));
    memset(lv, 0, sizeof(lv));
    c.L = L;
    c.k = k;
    for (i = 0; i < L->d; i++)
        if (i != k) dims[m++] = i;
    enum_levels(L, dims, m, 0, L->n - 1, 0, lv, chain_visit, &c);
    if (c.err) {
        free(c.chains);
        free(c.seg);
        return c.err;
    }
    if (c.nch > 1) qsort(c.chains, (size_t)c.nch, sizeof(sg_chain), chain_size_cmp);
    *chains = c.chains;
    *nchains = c.nch;
    *seg_off = c.seg;
    *nseg = c.nseg;
    return SG_OK;
}

/* ---- passes of several sweeps -------------------------------------------- */

/* nodes of the grid of dims k0..k0+g-1 with budget R */
static int64_t pass_nodes(const sg_layout *L, int k0, int g, int R)
{
    int64_t c[SG_MAX_LEVELS], t = 0;
    int i, s, l;
    for (s = 0; s <= R; s++) c[s] = s == 0;
    for (i = k0; i < k0 + g; i++)
        for (s = R; s >= 0; s--) {
            int64_t v = 0;
            for (l = 0; l <= s && l <= L->lim[i]; l++) v += c[s - l];
            c[s] = v;
        }
    for (s = 0; s <= R; s++) t += c[s] << s;
    return t;
}

int sg_layout_pass_dims(const sg_layout *L, int k0, int elem_bytes)
{
    const int most = L->d - k0 < 3 ? L->d - k0 : 3;
    int g, R;
    /* a single dim gains nothing over the single-dim sweep, except as the
     * rest of a grid that is otherwise done in passes */
    for (g = most; g >= (k0 > 0 ? 1 : 2); g--) {
        /* the largest unit's nodes: one CTA works through them, so three dims
         * only where that is short (n <= 6), two up to n = 10, and only where it
         * is a small part of the grid (d >= 5 or so) */
        const int64_t nodes = pass_nodes(L, k0, g, L->n - 1);
        int64_t elems = 0;
        if (nodes > (g == 3 ? SG_PASS3_NODES : SG_PASS_NODES) || 16 * nodes > L->N) continue;
        for (R = 1; R < L->n; R++) {
            const int64_t e = pass_nodes(L, k0, g, R) * sgk_unit_stride(L->n - 1 - R);
            if (e > elems) elems = e;
        }
        if (elems * elem_bytes <= (g == 1 ? SG_PASS1_BYTES : SG_UNIT_MAX_BYTES)) return g;
    }
    return 0;
}

void sg_layout_pass_free(sg_pass_host *p)
{
    free(p->units);
    free(p->offs);
    free(p->combos);
    free(p->nodes);
    free(p->combo_of);
    memset(p, 0, sizeof(*p));
}

typedef struct {
    const sg_layout *L;
    sg_pass_host *p;
    int k0, g;
    int64_t cap_u, cap_o;
    int err;
} unit_ctx;

static void unit_visit(void *vctx, int *lv, int sigma)
{
    unit_ctx *c = (unit_ctx *)vctx;
    const sg_layout *L = c->L;
    sg_pass_host *p = c->p;
    const int R = L->n - 1 - sigma;
    int i, m, lo = 0, nc;
    int64_t e;
    if (c->err || R < 1) return;
    nc = p->tables.ncombo[R];
    if (nc < 2) return; /* limits leave nothing to sweep */
    if (p->nunits == c->cap_u) {
        void *q;
        c->cap_u = c->cap_u ? 2 * c->cap_u : 1024;
        q = realloc(p->units, (size_t)c->cap_u * sizeof(sg_unit));
        if (!q) { c->err = SG_ERR_NOMEM; return; }
        p->units = (sg_unit *)q;
    }
    while (p->noffs + nc > c->cap_o) {
        void *q;
        c->cap_o = c->cap_o ? 2 * c->cap_o : 4096;
        q = realloc(p->offs, (size_t)c->cap_o * sizeof(uint32_t));
        if (!q) { c->err = SG_ERR_NOMEM; return; }
        p->offs = (uint32_t *)q;
    }
    for (m = c->k0 + c->g; m < L->d; m++) lo += lv[m];
    p->units[p->nunits].off = (uint32_t)p->noffs;
    p->units[p->nunits].R = (uint8_t)R;
    p->units[p->nunits].sigma = (uint8_t)sigma;
    p->units[p->nunits].lo = (uint8_t)lo;
    p->units[p->nunits].pad = 0;
    p->nunits++;
    for (i = 0; i < nc; i++) {
        for (m = 0; m < c->g; m++) lv[c->k0 + m] = p->combos[i].lv[m];
        p->offs[p->noffs++] = (uint32_t)sg_layout_subspace_offset(L, lv);
    }
    for (m = 0; m < c->g; m++) lv[c->k0 + m] = 0;
    i = nc - 1;
    e = ((int64_t)p->combos[i].node + ((int64_t)1 << p->combos[i].sum)) * sgk_unit_stride(sigma);
    if (e > p->max_elems) p->max_elems = e;
}

/* largest budgets first: their CTAs run longest */
static int unit_cmp(const void *a, const void *b)
{
    const sg_unit *x = (const sg_unit *)a, *y = (const sg_unit *)b;
    if (x->R != y->R) return x->R > y->R ? -1 : 1;
    return x->off < y->off ? -1 : (x->off > y->off);
}

/* the 1-D parent of index i at level j on one side: -1 at the boundary */
static int parent_of(int i, int j, int side, int *level)
{
    int m = i + side, tz = 0;
    if (m == 0 || m == (1 << j)) return -1;
    while (!((m >> tz) & 1)) tz++;
    *level = j - 1 - tz;
    return m >> (tz + 1);
}

int sg_layout_pass(const sg_layout *L, int k0, int g, sg_pass_host *p)
{
    int id[SG_MAX_LEVELS][SG_MAX_LEVELS][SG_MAX_LEVELS];
    int dims[SG_MAX_DIMS], lv[SG_MAX_DIMS], lim[3], m = 0, i, q, s, a, b, c;
    uint32_t fill[3][SG_MAX_LEVELS];
    sg_unit_tables *t = &p->tables;
    unit_ctx ctx;
    int64_t node = 0, total = 0;
    memset(p, 0, sizeof(*p));
    for (q = 0; q < 3; q++) {
        lim[q] = q < g ? L->lim[k0 + q] : 0;
        t->lmax[q] = lim[q];
    }
    /* combos by level sum */
    p->combos = (sg_unit_combo *)malloc(sizeof(sg_unit_combo) * SG_MAX_LEVELS * SG_MAX_LEVELS * SG_MAX_LEVELS);
    if (!p->combos) return SG_ERR_NOMEM;
    for (s = 0; s < L->n; s++) {
        for (a = 0; a <= s && a <= lim[0]; a++)
            for (b = 0; a + b <= s && b <= lim[1]; b++) {
                c = s - a - b;
                if (c > lim[2]) continue;
                id[a][b][c] = (int)p->ncombos;
                p->combos[p->ncombos].lv[0] = (uint8_t)a;
                p->combos[p->ncombos].lv[1] = (uint8_t)b;
                p->combos[p->ncombos].lv[2] = (uint8_t)c;
                p->combos[p->ncombos].sum = (uint8_t)s;
                p->combos[p->ncombos].node = (uint32_t)node;
                p->ncombos++;
                node += (int64_t)1 << s;
            }
        t->ncombo[s] = (int)p->ncombos;
        t->nnode[s] = (int)node;
    }
    if (node > SG_UNIT_NONE) return SG_ERR_RANGE;
    p->nall = node;
    p->combo_of = (uint16_t *)malloc(sizeof(uint16_t) * (size_t)node);
    if (!p->combo_of) return SG_ERR_NOMEM;
    for (m = 0; m < p->ncombos; m++)
        for (i = 0; i < 1 << p->combos[m].sum; i++) p->combo_of[p->combos[m].node + (uint32_t)i] = (uint16_t)m;
    /* lists of the points of level j in dim q, in node order (so by level sum) */
    for (q = 0; q < g; q++)
        for (i = 1; i <= lim[q]; i++) {
            uint32_t run = 0;
            t->first[q][i] = fill[q][i] = (uint32_t)total;
            for (s = 0; s < L->n; s++) {
                for (m = s ? t->ncombo[s - 1] : 0; m < t->ncombo[s]; m++)
                    if (p->combos[m].lv[q] == i) run += 1u << s;
                t->count[q][i][s] = (uint16_t)run;
            }
            total += run;
        }
    p->nnodes = total;
    p->nodes = (sg_unit_node *)malloc(sizeof(sg_unit_node) * (size_t)(total > 0 ? total : 1));
    if (!p->nodes) return SG_ERR_NOMEM;
    for (m = 0; m < p->ncombos; m++) {
        const sg_unit_combo *cb = &p->combos[m];
        for (q = 0; q < g; q++) {
            const int j = cb->lv[q];
            int below = 0, e, side;
            if (j < 1) continue;
            for (i = q + 1; i < g; i++) below += cb->lv[i]; /* index bits under dim q's */
            for (e = 0; e < 1 << cb->sum; e++) {
                const int ik = (e >> below) & ((1 << j) - 1), hi = e >> (below + j), lw = e & ((1 << below) - 1);
                sg_unit_node *out = &p->nodes[fill[q][j]++];
                out->node = (uint16_t)(cb->node + (uint32_t)e);
                out->pad = 0;
                for (side = 0; side < 2; side++) {
                    int pl = 0, pi = parent_of(ik, j, side, &pl), l3[3] = {cb->lv[0], cb->lv[1], cb->lv[2]};
                    uint16_t at = SG_UNIT_NONE;
                    if (pi >= 0) {
                        l3[q] = pl;
                        at = (uint16_t)(p->combos[id[l3[0]][l3[1]][l3[2]]].node +
                                        (uint32_t)((((hi << pl) | pi) << below) | lw));
                    }
                    if (side == 0) out->left = at;
                    else out->right = at;
                }
            }
        }
    }
    memset(&ctx, 0, sizeof(ctx));
    memset(lv, 0, sizeof(lv));
    ctx.L = L;
    ctx.p = p;
    ctx.k0 = k0;
    ctx.g = g;
    m = 0;
    for (i = 0; i < L->d; i++)
        if (i < k0 || i >= k0 + g) dims[m++] = i;
    enum_levels(L, dims, m, 0, L->n - 1, 0, lv, unit_visit, &ctx);
    if (ctx.err) return ctx.err;
    if (p->nunits > 1) qsort(p->units, (size_t)p->nunits, sizeof(sg_unit), unit_cmp);
    return SG_OK;
}

int64_t sg_layout_sweep_bytes(const sg_layout *L)
{
    int64_t bytes = 0;
    int k, g, s, a, b, c;
    for (k = 0; k < L->d; k += g > 0 ? g : 1) {
        g = sg_layout_pass_dims(L, k, 4);
        /* chains or units of two subspaces at least (8 bytes each), and an
         * offset per subspace */
        bytes += 8 * L->S;
        if (!g) continue;
        bytes += (int64_t)(g * sizeof(sg_unit_node) + 2) * pass_nodes(L, k, g, L->n - 1);
        for (s = 0; s < L->n; s++)
            for (a = 0; a <= s && a <= L->lim[k]; a++)
                for (b = 0; a + b <= s && b <= (g > 1 ? L->lim[k + 1] : 0); b++) {
                    c = s - a - b;
                    if (c <= (g > 2 ? L->lim[k + 2] : 0)) bytes += sizeof(sg_unit_combo);
                }
    }
    return bytes;
}

/* ---- evaluation (block) layout ------------------------------------------ */

static int lim_of(const sg_layout *L, int k) { return k >= 0 ? L->lim[k] : 0; }

void sg_layout_eval_sub(const sg_layout *L, int r, sg_eval_sub *sh)
{
    const int limA = lim_of(L, L->d - 2), limB = L->lim[L->d - 1];
    int a;
    uint32_t off = 0;
    memset(sh, 0, sizeof(*sh));
    sh->amax = r < limA ? r : limA;
    for (a = 0; a <= sh->amax; a++) {
        int rl = r - a < limB ? r - a : limB;
        sh->rowlen[a] = rl + 1;
        sh->aoff[a] = off;
        off += SG_POLE_SLOTS(rl) << a; /* 2^a poles */
    }
    sh->aoff[sh->amax + 1] = off;
}

void sg_layout_eval_shape(const sg_layout *L, int R, sg_eval_shape *sh)
{
    const int limC = lim_of(L, L->d - 3);
    int c;
    uint32_t off = 0;
    memset(sh, 0, sizeof(*sh));
    sh->R = R;
    sh->cmax = R < limC ? R : limC;
    for (c = 0; c <= sh->cmax; c++) {
        sg_eval_sub sub;
        sg_layout_eval_sub(L, R - c, &sub);
        sh->coff[c] = off;
        off += ((uint32_t)1 << c) * sub.aoff[sub.amax + 1];
    }
    sh->coff[sh->cmax + 1] = off;
}

/* Values of the block layout: every prefix level vector's cells times the
 * block size of its remaining budget. */
static int64_t block_layout_size(const sg_layout *L)
{
    const int np_dims = L->d >= 3 ? L->d - 3 : 0;
    int64_t sz[SG_MAX_DIMS + 1][SG_MAX_LEVELS];
    int k, R;
    for (R = 0; R < L->n; R++) {
        sg_eval_shape sh;
        sg_layout_eval_shape(L, R, &sh);
        sz[np_dims][R] = sh.coff[sh.cmax + 1];
    }
    for (k = np_dims - 1; k >= 0; k--)
        for (R = 0; R < L->n; R++) {
            int l;
            int64_t w = 0;
            for (l = 0; l <= R && l <= L->lim[k]; l++) w += sz[k + 1][R - l] << l;
            sz[k][R] = w;
        }
    return sz[0][L->n - 1];
}

int sg_layout_eval_tables(const sg_layout *L, sg_repack **repack, uint32_t **src, uint32_t *blk3, uint32_t *blk2)
{
    const int d = L->d;
    const int np_dims = d >= 3 ? d - 3 : 0; /* dims 0..d-4 form the prefix */
    int lv[SG_MAX_DIMS], k, s, R, b;
    int64_t pos, r = 0, q = 0;
    /* sz[k][R]: total block-layout size of the blocks (all cells) of the
     * level vectors over prefix dims k..np_dims-1 with sum <= R */
    int64_t sz[SG_MAX_DIMS + 1][SG_MAX_LEVELS];
    sg_eval_shape shape[SG_MAX_LEVELS];
    sg_eval_sub subs[SG_MAX_LEVELS];
    sg_repack *rp;
    uint32_t *so;
    for (R = 0; R < L->n; R++) {
        sg_layout_eval_shape(L, R, &shape[R]);
        sg_layout_eval_sub(L, R, &subs[R]);
        blk3[R] = shape[R].coff[shape[R].cmax + 1];
        blk2[R] = subs[R].aoff[subs[R].amax + 1];
        sz[np_dims][R] = blk3[R];
    }
    for (k = np_dims - 1; k >= 0; k--)
        for (R = 0; R < L->n; R++) {
            int l;
            int64_t w = 0;
            for (l = 0; l <= R && l <= L->lim[k]; l++) w += sz[k + 1][R - l] << l; /* 2^l cells of this dim */
            sz[k][R] = w;
        }
    if (sz[0][L->n - 1] != L->Nblk) return SG_ERR_STATE;
    rp = (sg_repack *)malloc((size_t)L->nrows * sizeof(sg_repack));
    so = (uint32_t *)malloc((size_t)L->S * sizeof(uint32_t));
    if (!rp || !so) {
        free(rp);
        free(so);
        return SG_ERR_NOMEM;
    }
    memset(lv, 0, sizeof(lv));
    for (s = 0; s < L->n; s++) {
        /* the level vectors of dims 0..d-2 with sum s, in the order of the
         * (d-1)-dimensional positions */
        const int64_t cnt = d >= 2 ? L->dp[d - 2][s] : s == 0;
        const int last = L->n - 1 - s < L->lim[d - 1] ? L->n - 1 - s : L->lim[d - 1];
        for (pos = 0; pos < cnt; pos++) {
            int c, a, rem = L->n - 1, sigma = 0, rest = s;
            int64_t base = 0, scale = 1, p = pos;
            const sg_eval_shape *sh;
            const sg_eval_sub *sub;
            for (k = d - 2; k >= 1; k--) {
                int level = 0;
                while (p >= L->dp[k - 1][rest - level]) p -= L->dp[k - 1][rest - level++];
                lv[k] = level;
                rest -= level;
            }
            if (d >= 2) lv[0] = rest;
            /* block-layout start of this prefix: the sizes of all prefixes
             * that precede it in the depth-first walk */
            for (k = 0; k < np_dims; k++) {
                int l;
                for (l = 0; l < lv[k]; l++) base += (sz[k + 1][rem - l] << l) * scale;
                scale <<= lv[k];
                rem -= lv[k];
                sigma += lv[k];
            }
            c = d >= 3 ? lv[d - 3] : 0;
            a = d >= 2 ? lv[d - 2] : 0;
            sh = &shape[L->n - 1 - sigma];
            sub = &subs[L->n - 1 - sigma - c];
            rp[r].src = (uint32_t)q;
            rp[r].dst = (uint32_t)base + sh->coff[c] + sub->aoff[a];
            rp[r].blk = sh->coff[sh->cmax + 1];
            rp[r].sub = sub->aoff[sub->amax + 1];
            rp[r].plen = SG_POLE_SLOTS(last);
            rp[r].c = (uint8_t)c;
            rp[r].a = (uint8_t)a;
            rp[r].L = (uint8_t)last;
            rp[r].s = (uint8_t)s;
            r++;
            /* subspace (lv, b): its position adds the vectors with a lower
             * level of dim d-1 */
            for (b = 0; b <= last; b++) {
                int64_t at = pos;
                int j;
                for (j = 0; d >= 2 && j < b; j++) at += L->dp[d - 2][s + b - j];
                so[q++] = (uint32_t)(L->plidx[s + b] + (at << (s + b)));
            }
        }
    }
    if (r != L->nrows || q != L->S) {
        free(rp);
        free(so);
        return SG_ERR_STATE;
    }
    *repack = rp;
    *src = so;
    return SG_OK;
}

/* ---- segments of the evaluation's sums ---------------------------------- */

int sg_layout_parts(const sg_layout *L)
{
    if (L->d < 4 || L->S < 4096) return 1;
    return L->S / 2048 < 8 ? (int)(L->S / 2048) : 8;
}

int sg_layout_segs(const sg_layout *L)
{
    const int parts = sg_layout_parts(L);
    if (L->d < 4) return 1;
    if (parts > 1) return parts * SG_SEG_PER_PART;
    if (L->S < 2 * SG_SEG_SUBSPACES) return 1;
    return L->S / SG_SEG_SUBSPACES < SG_SEG_PER_PART ? (int)(L->S / SG_SEG_SUBSPACES) : SG_SEG_PER_PART;
}

int64_t sg_layout_seg_words(const sg_layout *L)
{
    const int nseg = sg_layout_segs(L);
    return nseg > 1 ? (int64_t)(L->d - 2) * L->n + nseg + 1 : 0;
}

/* rows (c, a) of the innermost dims with c + a <= R, in limits */
static double block_rows(const sg_layout *L, int R)
{
    const int lc = L->lim[L->d - 3], la = L->lim[L->d - 2];
    double cnt = 0.0;
    int c;
    for (c = 0; c <= R && c <= lc; c++) cnt += (R - c < la ? R - c : la) + 1;
    return cnt;
}

#define SG_BLOCK_OVERHEAD 2.0 /* per-block walk cost in rows */

int sg_layout_seg_table(const sg_layout *L, const uint32_t *blk3, uint32_t *table)
{
    const int d = L->d, n = L->n, nseg = sg_layout_segs(L);
    /* deepest loop whose iterations a segment may start at: the dims from
     * d-4 on run as one unit (d = 4: its only loop) */
    const int deep = d == 4 ? 0 : d - 5;
    uint32_t *bounds = table + (d - 2) * n;
    double *W;
    int K, b, l, j;
    if (nseg <= 1) return SG_ERR_ARG;
    W = (double *)malloc(sizeof(double) * (size_t)(d - 2) * (size_t)n);
    if (!W) return SG_ERR_NOMEM;
    for (b = 0; b < n; b++) {
        W[(d - 3) * n + b] = block_rows(L, b) + SG_BLOCK_OVERHEAD;
        table[(d - 3) * n + b] = blk3[b] << (n - 1 - b);
    }
    for (K = d - 4; K >= 0; K--)
        for (b = 0; b < n; b++) {
            double w = 0.0;
            uint64_t ext = 0;
            for (l = 0; l <= b && l <= L->lim[K]; l++) {
                w += W[(K + 1) * n + b - l];
                ext += table[(K + 1) * n + b - l];
            }
            W[K * n + b] = w;
            table[K * n + b] = (uint32_t)ext;
        }
    bounds[0] = 0;
    bounds[nseg] = table[n - 1];
    for (j = 1; j < nseg; j++) {
        /* descend to the unit holding work position j/nseg of the total; the
         * segment starts where the unit does.  Units: iterations of the loop
         * at depth `deep`, and whole nodes of that depth with a budget the
         * kernels may unroll (SG_SEG_UNIT_BUDGET) */
        const double t = W[n - 1] * j / nseg;
        double acc = 0.0;
        uint32_t at = 0;
        K = 0;
        b = n - 1;
        while (K <= deep && !(K == deep && d > 4 && b <= SG_SEG_UNIT_BUDGET)) {
            const int lmax = b < L->lim[K] ? b : L->lim[K];
            for (l = 0; l < lmax; l++) {
                const double w = W[(K + 1) * n + b - l];
                if (acc + w > t) break;
                acc += w;
                at += table[(K + 1) * n + b - l];
            }
            K++;
            b -= l;
        }
        bounds[j] = at < bounds[j - 1] ? bounds[j - 1] : at;
    }
    free(W);
    return SG_OK;
}
