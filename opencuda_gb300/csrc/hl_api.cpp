/*
 * hl_api.cpp -- the C ABI: handle, workspace and the stage pipeline.
 *
 * hl_plain is HoughLine::houghLine (okano_3_0/HoughLine.cu:635-955) without
 * its per-call cudaMalloc/cudaFree and without the two accumulator-sized
 * device->host copies: four kernels run back to back on the caller's stream
 *   compact (a) -> vote (b) -> peaks (c1) -> finalize (c2)
 * and one small transfer brings back a header plus linesmax LineParam
 * records.  The workspace is owned by the handle and grows only when a
 * larger ROI arrives.
 */
#include <cuda_runtime.h>

#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <functional>
#include <queue>
#include <new>
#include <vector>

#include "hl_internal.h"
#include "hl_cnn.h"
#include "hl_proposal.h"
#include "hl_window.h"

#ifndef M_PI
#error "M_PI required: numtheta = (int)(M_PI / detheta)"
#endif

struct hl_batch_ws;   /* batched-path workspace (hl_batch*) */
/* a handle's accumulator: anything; zero in the rows that the plan's votes never
 * reach; all zero */
enum { ACC_ANY = 0, ACC_UNREACHED, ACC_ZERO };

struct hl_handle {
    hl_params p;
    int T, Tp;
    int device;
    int sms;
    float *d_cos, *d_sin;
    float *h_cos, *h_sin;    /* host copies of the table */

    uint32_t *d_pts;
    size_t cap_pts;
    unsigned long long *d_tile_state;
    int *d_tile_off;
    size_t cap_tiles;
    int32_t *d_acc;
    size_t cap_acc;
    unsigned long long *d_keys;
    size_t cap_keys;
    int32_t *d_aux;          /* tight / reference layout staging */
    size_t cap_aux;
    unsigned char *d_result; /* hl_result_hdr + lines */
    size_t cap_result;
    unsigned char *h_result; /* pinned mirror */
    /* counters: [0] ncand, [1] status, [2] points, [3] ticket, [4] bbox
     * ticket, [8] realLine, [9] vote work, [10] peak candidates */
    int *d_counters;
    int4 *d_bbox;            /* partial boxes of a coordinate list */
    int *h_bbox;             /* its box (pinned; the kernel writes it) */

    unsigned ticket_base;
    unsigned epoch;
    int win_rows_override, threads_override;
    int last_launches;

    /* the vote plan of the last geometry (reused while it is the same) and
     * the persistent-CTA counter base */
    struct vote_plan *plan;
    int plan_w, plan_h, plan_R, plan_T, plan_cap, plan_thr;
    int acc_state;           /* what is known of d_acc (ACC_*) */
    int cand_par;            /* the noted candidates' counter: [10 + cand_par] */
    double plan_detheta, plan_derho;
    unsigned char *d_plan;   /* items, merge blocks, slab list */
    size_t cap_plan;
    unsigned char *h_plan;   /* its pinned staging copy ... */
    size_t cap_hplan;
    cudaEvent_t plan_read;   /* ... and the last upload's end */
    int plan_event;
    unsigned char *d_scratch;
    size_t cap_scratch;
    unsigned long long *d_cand;   /* noted peak candidates */
    size_t cap_cand;
    /* HoughCircle: candidate keys, [ncand, status] counters, results; the
     * workspace of circle batches */
    struct hl_cb_ws *cb;
    int *d_ctab;             /* the circles' offsets (hl_circle_table_kernel) */
    uint32_t *d_cbits;       /* an image's edge map */
    size_t cap_cbits;
    unsigned long long *d_ckeys;
    int *d_ccnt;
    unsigned char *d_cres;
    unsigned char *h_cres;
    unsigned work_base;

    /* batched path: workspace, CUDA-graph switch; whether the last
     * asynchronous call was a batch (hl_last_status reads its status) */
    hl_batch_ws *bw;
    hl_batch_ws *bw_fb;     /* the proposal path's fall-back batches */
    struct hl_prop_ws *pw;  /* the proposal path's own buffers */
    int batch_graph;
    int last_batch;

    /* per-stage CUDA-event timing (hl_profile) */
    int prof;
    int prof_open;
    int prof_used;
    cudaEvent_t *prof_ev;   /* HL_PROF_MAX x HL_NSTAGE+1 */
};

#define HL_NSTAGE 4
#define HL_PROF_MAX 512

/* Record the event that closes stage `st` (0 = before the first stage). */
static void prof_mark(hl_handle *h, int st, cudaStream_t s)
{
    if (!h->prof || !h->prof_ev || h->prof_used >= HL_PROF_MAX)
        return;
    if (st == 0)
        h->prof_open = 1;
    else if (!h->prof_open)
        return;   /* a call that did not start at stage (a) */
    cudaEventRecord(h->prof_ev[h->prof_used * (HL_NSTAGE + 1) + st], s);
    if (st == HL_NSTAGE) {
        h->prof_used++;
        h->prof_open = 0;
    }
}

/* An error is reported once: the runtime keeps a failed call's as the last error,
 * which the check after the next launch would take for that launch's. */
static int map_err(cudaError_t e)
{
    if (e == cudaSuccess)
        return HL_NO_ERROR;
    cudaGetLastError();
    if (e == cudaErrorMemoryAllocation)
        return HL_OUT_OF_MEM;
    return HL_CUDA_ERROR;
}

#define CK(call)                                  \
    do {                                          \
        cudaError_t e__ = (call);                 \
        if (e__ != cudaSuccess)                   \
            return map_err(e__);                  \
    } while (0)

static int grow(void **ptr, size_t *cap, size_t need_bytes)
{
    if (*cap >= need_bytes && *ptr)
        return HL_NO_ERROR;
    size_t nb = std::max(need_bytes, (size_t)256);
    nb = nb + nb / 4;   /* headroom for the next, slightly larger ROI */
    if (*ptr) {
        cudaFree(*ptr);   /* synchronises: nothing in flight uses it */
        *ptr = nullptr;
        *cap = 0;
    }
    cudaError_t e = cudaMalloc(ptr, nb);
    if (e != cudaSuccess) {
        *ptr = nullptr;
        return map_err(e);
    }
    *cap = nb;
    return HL_NO_ERROR;
}

static int grow_host(unsigned char **ptr, size_t *cap, size_t need)
{
    if (*cap >= need && *ptr)
        return HL_NO_ERROR;
    size_t nb = std::max(need, (size_t)4096);
    nb += nb / 4;
    if (*ptr)
        cudaFreeHost(*ptr);
    *ptr = nullptr;
    *cap = 0;
    CK(cudaMallocHost(ptr, nb));
    *cap = nb;
    return HL_NO_ERROR;
}

static int check_params(const hl_params *p)
{
    if (!(p->detheta > 0.0) || !(p->derho > 0.0))
        return HL_INVALID_DATA;
    double t = M_PI / p->detheta;
    if (!(t >= 1.0) || t > 65536.0)
        return HL_INVALID_DATA;
    return HL_NO_ERROR;
}

static int build_table(hl_handle *h)
{
    h->T = (int)(M_PI / h->p.detheta);          /* okano_3_0/HoughLine.cu:671 */
    h->Tp = (h->T + HL_SLICE - 1) / HL_SLICE * HL_SLICE;
    if (h->d_cos)
        cudaFree(h->d_cos);
    if (h->d_sin)
        cudaFree(h->d_sin);
    h->d_cos = h->d_sin = nullptr;
    CK(cudaMalloc(&h->d_cos, sizeof(float) * h->Tp));
    CK(cudaMalloc(&h->d_sin, sizeof(float) * h->Tp));
    CK(hl_launch_trig(h->d_cos, h->d_sin, h->T, h->Tp, h->p.detheta, 0));
    free(h->h_cos);
    free(h->h_sin);
    h->h_cos = (float *)malloc(sizeof(float) * h->Tp);
    h->h_sin = (float *)malloc(sizeof(float) * h->Tp);
    if (!h->h_cos || !h->h_sin)
        return HL_OUT_OF_MEM;
    CK(cudaMemcpyAsync(h->h_cos, h->d_cos, sizeof(float) * h->Tp, cudaMemcpyDeviceToHost, 0));
    CK(cudaMemcpyAsync(h->h_sin, h->d_sin, sizeof(float) * h->Tp, cudaMemcpyDeviceToHost, 0));
    CK(cudaStreamSynchronize(0));
    return HL_NO_ERROR;
}

extern "C" int hl_create(hl_handle **out, const hl_params *params)
{
    if (!out)
        return HL_NULL_POINTER;
    *out = nullptr;
    hl_params p;
    if (params) {
        p = *params;
    } else {   /* okano_3_0/HoughLine.h:120-124 */
        p.detheta = M_PI / 180;
        p.derho = 1.0;
        p.threshold = 90;
        p.thresang = (float)(M_PI / 180 * 5.0f);
        p.thresdis = 50;
    }
    int rc = check_params(&p);
    if (rc != HL_NO_ERROR)
        return rc;
    hl_handle *h = new (std::nothrow) hl_handle();
    if (!h)
        return HL_OUT_OF_MEM;
    memset(h, 0, sizeof(*h));
    h->p = p;
    cudaError_t e = cudaGetDevice(&h->device);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount,
                                   h->device);
    if (e == cudaSuccess)
        e = cudaMalloc(&h->d_counters, 16 * sizeof(int));
    if (e == cudaSuccess)
        e = cudaMemset(h->d_counters, 0, 16 * sizeof(int));
    if (e != cudaSuccess) {
        hl_destroy(h);
        return map_err(e);
    }
    rc = build_table(h);
    if (rc != HL_NO_ERROR) {
        hl_destroy(h);
        return rc;
    }
    *out = h;
    return HL_NO_ERROR;
}

static void batch_free(hl_handle *h);
static void circle_batch_free(hl_handle *h);
static void plan_free(struct vote_plan *p);

extern "C" int hl_destroy(hl_handle *h)
{
    if (!h)
        return HL_NULL_POINTER;
    batch_free(h);
    circle_batch_free(h);
    plan_free(h->plan);
    void *ptrs[] = {h->d_cos, h->d_sin, h->d_pts, h->d_tile_state,
                    h->d_tile_off, h->d_acc, h->d_keys, h->d_aux,
                    h->d_result, h->d_counters, h->d_plan, h->d_scratch, h->d_cand,
                    h->d_ckeys, h->d_ccnt, h->d_cres, h->d_bbox, h->d_ctab,
                    h->d_cbits};
    for (void *q : ptrs)
        if (q)
            cudaFree(q);
    if (h->h_result)
        cudaFreeHost(h->h_result);
    if (h->h_cres)
        cudaFreeHost(h->h_cres);
    if (h->h_bbox)
        cudaFreeHost(h->h_bbox);
    if (h->h_plan)
        cudaFreeHost(h->h_plan);
    if (h->plan_event)
        cudaEventDestroy(h->plan_read);
    free(h->h_cos);
    free(h->h_sin);
    if (h->prof_ev) {
        for (int i = 0; i < HL_PROF_MAX * (HL_NSTAGE + 1); i++)
            cudaEventDestroy(h->prof_ev[i]);
        free(h->prof_ev);
    }
    delete h;
    return HL_NO_ERROR;
}

extern "C" int hl_profile(hl_handle *h, int enable)
{
    if (!h)
        return HL_NULL_POINTER;
    if (enable && !h->prof_ev) {
        int n = HL_PROF_MAX * (HL_NSTAGE + 1);
        h->prof_ev = (cudaEvent_t *)calloc((size_t)n, sizeof(cudaEvent_t));
        if (!h->prof_ev)
            return HL_OUT_OF_MEM;
        for (int i = 0; i < n; i++)
            CK(cudaEventCreate(&h->prof_ev[i]));
    }
    h->prof = enable ? 1 : 0;
    h->prof_used = 0;
    return HL_NO_ERROR;
}

extern "C" int hl_profile_read(hl_handle *h, double *stage_ms, int *calls)
{
    if (!h || !stage_ms || !calls)
        return HL_NULL_POINTER;
    for (int s = 0; s < HL_NSTAGE; s++)
        stage_ms[s] = 0.0;
    *calls = h->prof_used;
    for (int c = 0; c < h->prof_used; c++) {
        cudaEvent_t *e = &h->prof_ev[c * (HL_NSTAGE + 1)];
        CK(cudaEventSynchronize(e[HL_NSTAGE]));
        for (int s = 0; s < HL_NSTAGE; s++) {
            float ms = 0.f;
            CK(cudaEventElapsedTime(&ms, e[s], e[s + 1]));
            stage_ms[s] += ms;
        }
    }
    h->prof_used = 0;
    return HL_NO_ERROR;
}

extern "C" int hl_set_params(hl_handle *h, const hl_params *params)
{
    if (!h || !params)
        return HL_NULL_POINTER;
    int rc = check_params(params);
    if (rc != HL_NO_ERROR)
        return rc;
    bool retable = params->detheta != h->p.detheta;
    h->p = *params;
    return retable ? build_table(h) : HL_NO_ERROR;
}

extern "C" int hl_get_params(const hl_handle *h, hl_params *params)
{
    if (!h || !params)
        return HL_NULL_POINTER;
    *params = h->p;
    return HL_NO_ERROR;
}

static void layout(const hl_handle *h, double extent, int *rho_min, int *R)
{
    int d = (int)floor(extent / h->p.derho + 0.5);
    *rho_min = -d;
    *R = 2 * d + 1;
}

extern "C" int hl_geometry(const hl_handle *h, int w, int hh, hl_geom *g)
{
    if (!h || !g)
        return HL_NULL_POINTER;
    if (w <= 0 || hh <= 0 || w > HL_MAX_SIDE || hh > HL_MAX_SIDE)
        return HL_INVALID_DATA;
    g->numtheta = h->T;
    g->theta_pad = h->Tp;
    layout(h, sqrt((double)w * w + (double)hh * hh), &g->rho_min, &g->numrho);
    /* okano_3_0/HoughLine.cu:670 */
    g->ref_numrho = (int)((double)(int)((w + hh) * 2 + 1) / h->p.derho);
    g->tiles_x = (w + HL_TILE_W - 1) / HL_TILE_W;
    g->tiles_y = (hh + HL_TILE_H - 1) / HL_TILE_H;
    if ((double)g->numrho * h->Tp >= 2147483647.0)
        return HL_OP_OVERFLOW;
    return HL_NO_ERROR;
}

extern "C" int hl_trig_table(hl_handle *h, float *cos_host, float *sin_host)
{
    if (!h || !cos_host || !sin_host)
        return HL_NULL_POINTER;
    CK(cudaMemcpy(cos_host, h->d_cos, sizeof(float) * h->T,
                  cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(sin_host, h->d_sin, sizeof(float) * h->T,
                  cudaMemcpyDeviceToHost));
    return HL_NO_ERROR;
}

extern "C" int hl_set_vote_shape(hl_handle *h, int window_rows, int threads)
{
    if (!h)
        return HL_NULL_POINTER;
    if (window_rows < 0 || threads < 0 || threads > 1024 || (threads & 31))
        return HL_INVALID_DATA;
    if (window_rows > 65535 || (threads > 0 && threads < 64))
        return HL_INVALID_DATA;   /* rows above the shared-memory limit are clamped */
    h->win_rows_override = window_rows;
    h->threads_override = threads;
    return HL_NO_ERROR;
}

extern "C" int hl_last_launch_count(const hl_handle *h)
{
    return h ? h->last_launches : 0;
}

/* ---- the vote plan ---------------------------------------------------------
 * Every image's theta slices are voted in regions, rectangles of compaction
 * tiles whose rho range over the slice fits a window in shared memory
 * (hl_vote_item).  A region's rows are its width times max|cos| plus its
 * height times max|sin| over the slice, so slices near an axis take long
 * regions across it.  The number of regions is at least what the rows need and
 * what spreads the launch's work over the CTAs (weight cap); among the grids
 * with enough of them the one that stores the fewest rows is taken.  Weights
 * are in pixels; a row of a window costs about HL_ROW_PIXELS of them (its
 * clearing, storing and merging against votes at the 2-3% of edge pixels that
 * maps hold).  Items go heaviest first; those that a list schedule starts in
 * the last 40% of the launch are halved, so the CTAs finish together. */
/* Rows: 24 or 160 pixels change a 4096 x 4096 image, T = 720, by less than 0.3 us,
 * 160 cost 64 cells of 256 x 256 10 us of 82. */
#define HL_ROW_PIXELS 64.0
/* Items per CTA the plan aims at.  More balance better, fewer store and merge
 * less: 1, 2, 3, 5 a CTA take 151.5, 147.2, 150.2, 153.2 us at 4096 x 4096, T =
 * 720, and 1036, 993, 1005, 1007 us in a proposal batch of 32 x 2048 x 2048. */
#define HL_PLAN_SHARE 2.0
/* No region below this for balance alone: a region's own start and its slab
 * then cost more than its votes.  1913 x 1077, T = 360: 64 K, 128 K, 192 K pixels
 * 45.6, 45.5, 43.1 us; 2048 x 2048, T = 360, lines drawn: 72.6, 73.6, 67.9 us. */
#define HL_MIN_REGION (192.0 * 1024.0)
/* A block may also be voted in windows: an item votes the image's points that may
 * reach its rows, and each window is final.  It needs no slabs and no merge, but
 * tests every vote and votes a point once a window that its tile may reach.  It is
 * the form for rho steps below 1, whose regions get small and store many rows, and
 * for launches too small to be worth a merge.  Windows that outweigh a CTA's share
 * are split into parts of their points, which go through slabs like regions.
 * The form is chosen by estimates in pixels as above.  A tested vote costs
 * HL_WINDOW_VOTE plain ones, an item's start and end HL_ITEM_PIXELS, a row of a slab
 * HL_SLAB_PIXELS more than another row, a merge launch HL_MERGE_PIXELS: fitted to
 * single images and batches of 512 x 512 to 4096 x 4096 at steps 1 to 0.05 in every
 * form.  At rho steps from 1 on only launches of less than HL_SMALL_PIXELS and two
 * blocks a CTA are looked at: in others regions win.
 * T = 180, a call by fixed windows of rows, which this replaced / by regions alone /
 * now: 16 images of 1000 x 900, step 0.1 229 / 1368 / 174 us, 0.05 380 / 2088 / 260,
 * 0.25 149 / 217 / 126; one of 2048 x 2048, 0.1 94 / 362 / 102, 0.05 141 / 467 / 108;
 * 512 x 512, 0.1 45 / 171 / 45; 16 of 512 x 512, step 1 58 / 66 / 58. */
#define HL_WINDOW_VOTE 1.7
#define HL_ITEM_PIXELS 120e3
#define HL_SLAB_PIXELS 100.0
#define HL_MERGE_PIXELS 60e3
#define HL_SMALL_PIXELS 400e3

struct vote_plan {
    std::vector<hl_vote_item> items;
    std::vector<hl_merge_block> blocks;
    std::vector<hl_slab> slabs;
    long long scratch_units;   /* row groups of slabs */
    unsigned chunks;           /* of a merge launch */
    int part16, win_rows, exact, win;
    /* the blocks' items add to the accumulator instead of going through slabs:
     * where these would take more than HL_MAX_SCRATCH and twice the accumulators
     * (images of 32 K and more a side, or a handful of angles: a slab's column groups
     * are as tall as their thetas lie apart), or could not be allocated.  Dense: the
     * accumulator is cleared before and scanned after */
    int add;
};
#define HL_MAX_SCRATCH (1LL << 30)
static size_t plan_scratch(const vote_plan &p)
{
    return (size_t)std::max(p.scratch_units, 1LL) * (p.part16 ? 64 : 128);
}
static void plan_free(vote_plan *p) { delete p; }

struct plan_img {
    int w, h, R, rho_min;
};

/* max|cos| and max|sin| of a slice's thetas times irho, with a little slack
 * for the vote rule's floats */
struct slice_ext {
    double c, s;
};

static void slice_extents(const hl_handle *h, std::vector<slice_ext> &ext)
{
    const double irho = 1.0 / h->p.derho;
    const int slices = h->Tp / HL_SLICE;
    ext.assign((size_t)slices, {0.0, 0.0});
    for (int k = 0; k < h->T; k++) {
        slice_ext &e = ext[(size_t)(k / HL_SLICE)];
        e.c = std::max(e.c, fabs((double)h->h_cos[k]) * irho * (1.0 + 1e-6));
        e.s = std::max(e.s, fabs((double)h->h_sin[k]) * irho * (1.0 + 1e-6));
    }
}

/* rows a region of gw x gh pixels needs over a slice (its range, both ends,
 * truncation and rounding) */
static double region_rows(const slice_ext &e, double gw, double gh)
{
    return (gw - 1.0) * e.c + (gh - 1.0) * e.s + 4.0;
}

struct plan_region {
    double wt;
    hl_vote_item it;
    int blk;
};

/* the grid of regions of one (image, slice): nx x ny; false where not even a tile's
 * rows fit a window */
static bool best_grid(const slice_ext &e, int w, int hh, int cap, double n_min, int *bx, int *by)
{
    const int tx = (w + HL_TILE_W - 1) / HL_TILE_W, ty = (hh + HL_TILE_H - 1) / HL_TILE_H;
    double best = 1e300;
    bool found = false;
    for (int nx = 1; nx <= tx; nx++) {
        const int gtx = (tx + nx - 1) / nx;
        if (nx > 1 && gtx == (tx + nx - 2) / (nx - 1))
            continue;   /* no narrower than with one column less */
        const double gw = std::min(gtx * HL_TILE_W, w);
        const double left = cap - 4.0 - (gw - 1.0) * e.c;
        if (left < 0.0)
            continue;
        /* tile rows a region may have */
        double tr = e.s > 0.0 ? floor((left / e.s + 1.0) / HL_TILE_H) : ty;
        if (tr < ty && hh <= HL_TILE_H && (hh - 1.0) * e.s <= left)
            tr = ty;
        if (nx > 1)
            tr = std::min(tr, (double)HL_VOTE_RUNS);
        if (tr < 1.0)
            continue;
        const int need_y = (int)ceil(ty / std::min(tr, (double)ty));
        const int ny = std::min(ty, std::max(need_y, (int)ceil(n_min / nx)));
        const double gh = std::min(((ty + ny - 1) / ny) * HL_TILE_H, hh);
        const double cost = (double)nx * ny * (region_rows(e, gw, gh) + 64.0);
        if (cost < best) {
            best = cost;
            *bx = nx;
            *by = ny;
            found = true;
        }
        if (nx > 4.0 * n_min + 8 && found)
            break;
    }
    return found;
}

/* The band of rows of one (image, slice) that windows share out, and what
 * hl_vote_item needs of it.  Relative to the centre's at the same theta a point's rho
 * is u cos d + v sin d, u and v its distances from the centre across and along the
 * middle theta's lines, d the angle to the middle. */
struct plan_band {
    int first;                /* off0 of the first window; the last one ends at -first */
    double out, tang;         /* pixels that a window's ends are moved outwards */
    double a, b, reach;       /* half widths of u's two parts; tang times the mean |v| */
};
static plan_band block_band(const hl_handle *h, int w, int hh, int sl)
{
    const int k0 = sl * HL_SLICE, k1 = std::min(k0 + HL_SLICE, h->T) - 1;
    const int km = std::min(k0 + HL_SLICE / 2, h->T - 1);
    const double irho = 1.0 / h->p.derho;
    const double x = 0.5 * w, y = 0.5 * hh;
    double half = 0.0, tile = 0.0;   /* pixels across that the image and a tile reach */
    for (int k = k0; k <= k1; k++) {
        const double c = fabs((double)h->h_cos[k]), s = fabs((double)h->h_sin[k]);
        half = std::max(half, x * c + y * s);
        tile = std::max(tile, 0.5 * HL_TILE_W * c + 0.5 * HL_TILE_H * s);
    }
    /* rows for the centre's floor, the votes' truncation, floats */
    const double slack = 4.0 + sqrt(4.0 * (x * x + y * y)) * irho * (1.0 / (1 << 19));
    const double d = std::max(k1 - km, km - k0) * h->p.detheta;
    const double c = fabs((double)h->h_cos[km]), s = fabs((double)h->h_sin[km]);
    plan_band p;
    p.first = -(int)ceil(half * irho + slack);
    /* the curvature: a tile's centre lies up to a tile outside the image */
    p.out = tile + (1.0 - cos(std::min(d, M_PI))) * ((x + HL_TILE_W) * c + (y + HL_TILE_H) * s) +
            2.0 + slack * h->p.derho;
    p.tang = d < 0.5 * M_PI ? sin(d) : 1.0;
    p.a = x * c;
    p.b = y * s;
    p.reach = p.tang * 0.5 * (x * s + y * c);
    return p;
}
/* its windows of at most cap rows: their number; *rows: rows of one */
static int band_windows(const plan_band &p, int cap, int *rows)
{
    const int total = 1 - 2 * p.first, n = (total + cap - 1) / cap;
    *rows = (total + n - 1) / n;
    return n;
}

/* the part of a rectangle's area that lies below u = v: u is the sum of two uniform
 * distances, in [-a, a] and [-b, b] */
static double area_below(double a, double b, double v)
{
    a = std::max(a, 1e-3);
    b = std::max(b, 1e-3);
    const auto sq = [](double t) { return t > 0.0 ? t * t : 0.0; };
    return (sq(v + a + b) - sq(v + a - b) - sq(v - a + b) + sq(v - a - b)) / (8.0 * a * b);
}

/* The item of a whole w x hh image whose range exceeds the window, voted with a
 * sliding window; false where one window holds it or sliding cannot.  A point's
 * rho relative to the centre's differs from its tile centre's at the middle
 * theta by at most the tile's half diagonal (66) and the centre distance times
 * the angle to the middle (16 steps at most), so a band of adv rows needs adv +
 * 2 e rows; the window moves by adv, at least half of itself, so that moving
 * the rest down does not overlap. */
static bool slide_item(const hl_handle *h, const slice_ext &e, int w, int hh, int sl, int cap,
                       hl_vote_item *it)
{
    const int tx = (w + HL_TILE_W - 1) / HL_TILE_W, ty = (hh + HL_TILE_H - 1) / HL_TILE_H;
    const double irho = 1.0 / h->p.derho;
    if (region_rows(e, w, hh) <= cap || ty > HL_VOTE_RUNS || irho > 4.0)
        return false;
    const double lx = 0.5 * w + HL_TILE_W, ly = 0.5 * hh + HL_TILE_H;
    const double dist = sqrt(lx * lx + ly * ly) * irho;
    const int err = (int)ceil(66.0 * irho + dist * 16.0 * h->p.detheta + dist * 1e-5) + 4;
    const int adv = (cap - 2 * err - 4) / 4 * 4;
    if (2 * adv < cap)
        return false;
    const int km = std::min(sl * HL_SLICE + HL_SLICE / 2, h->T - 1);
    const double half = ceil(lx * fabs((double)h->h_cos[km]) * irho +
                             ly * fabs((double)h->h_sin[km]) * irho) + 2.0;
    memset(it, 0, sizeof(*it));
    it->slice = sl;
    it->tx = tx << 16;
    it->ty = ty << 16;
    it->slab = -1;
    it->nseg = (int)ceil(2.0 * half / adv);
    it->adv = adv;
    it->off0 = -(int)half - err;
    it->half = (float)half;
    return it->nseg > 1;
}

/* column group g holds the rows r0 to r1 of R4 groups of four */
static void slab_rows(hl_slab *sl, int g, double r0, double r1, int R4)
{
    const int b = (int)std::min(std::max(floor(r0 / 4.0), 0.0), (double)R4);
    const int e = (int)std::min(std::max(floor(r1 / 4.0) + 1.0, (double)b), (double)R4);
    sl->b[g] = b;
    sl->n[g] = e - b;
    if (e > b) {
        sl->lo = std::min(sl->lo, b);
        sl->hi = std::max(sl->hi, e);
    }
}

/* 1 - cos(half the span) of the eight columns from k0 on */
static double slab_bend(const hl_handle *h, int k0)
{
    const int k1 = std::min(k0 + 7, h->T - 1);
    return 1.0 - cos(std::min(0.5 * (k1 - std::min(k0, k1)) * h->p.detheta, M_PI));
}

/* The rows that the votes of an item's four column groups can fall into, in
 * groups of four rows (sl's b, n, lo and hi).  A corner's rho is a sinusoid over
 * the group's thetas: no lower than at its ends less the distance times 1 -
 * cos(half the span) (bend, of the slice's groups), and as much higher; a row and
 * 2^-20 of the value more for the vote rule's floats. */
static void slab_groups(const hl_handle *h, const plan_img &im, const hl_vote_item &it, int x1,
                        int y1, const double *bend, hl_slab *sl)
{
    const double irho = 1.0 / h->p.derho;
    const int R4 = (im.R + 3) / 4;
    const double xs[2] = {(double)((it.tx & 0xffff) * HL_TILE_W), x1 - 1.0};
    const double ys[2] = {(double)((it.ty & 0xffff) * HL_TILE_H), y1 - 1.0};
    const double far = sqrt(xs[1] * xs[1] + ys[1] * ys[1]) * irho;
    sl->lo = 0x7fffffff;
    sl->hi = 0;
    for (int g = 0; g < 4; g++) {
        /* columns past the last theta vote like it, and are cleared alike */
        const int k0 = std::min(it.slice * HL_SLICE + 8 * g, h->T - 1);
        const int k1 = std::min(it.slice * HL_SLICE + 8 * g + 7, h->T - 1);
        double lo = 1e300, hi = -1e300;
        for (int e = 0; e < 8; e++) {
            const int k = e & 4 ? k1 : k0;
            const double v = (xs[e & 1] * (double)h->h_cos[k] +
                              ys[(e >> 1) & 1] * (double)h->h_sin[k]) * irho;
            lo = std::min(lo, v);
            hi = std::max(hi, v);
        }
        const double slack = far * bend[g] + far * (1.0 / (1 << 20)) + 1.0;
        slab_rows(sl, g, floor(lo - slack) - im.rho_min, ceil(hi + slack) - im.rho_min, R4);
    }
}

/* the same for an item of one window: the rows that its columns hold (a row and 2^-20
 * of the value more for the device's floats) */
static void window_groups(const hl_handle *h, const plan_img &im, const hl_vote_item &it,
                          hl_slab *sl)
{
    const double irho = 1.0 / h->p.derho, x = 0.5 * (im.w - 1), y = 0.5 * (im.h - 1);
    const double slack = sqrt(x * x + y * y) * irho * (1.0 / (1 << 20)) + 2.0;
    const int R4 = (im.R + 3) / 4;
    sl->lo = 0x7fffffff;
    sl->hi = 0;
    for (int g = 0; g < 4; g++) {
        double lo = 1e300, hi = -1e300;
        for (int c = 0; c < 8; c++) {
            const int k = std::min(it.slice * HL_SLICE + 8 * g + c, h->T - 1);
            const double v = (x * (double)h->h_cos[k] + y * (double)h->h_sin[k]) * irho;
            lo = std::min(lo, v);
            hi = std::max(hi, v);
        }
        slab_rows(sl, g, floor(lo - slack) + it.off0 - im.rho_min,
                  ceil(hi + slack) + it.off0 + it.adv - im.rho_min, R4);
    }
}

/* pixels of window j of rows rows */
static double window_weight(const hl_handle *h, const plan_band &p, double area, int j, int rows)
{
    const double lo = (p.first + (double)j * rows) * h->p.derho - p.out - p.reach;
    const double hi = (p.first + (double)(j + 1) * rows) * h->p.derho + p.out + p.reach;
    return area * HL_WINDOW_VOTE * (area_below(p.a, p.b, hi) - area_below(p.a, p.b, lo)) +
           HL_ROW_PIXELS * rows;
}
/* parts of a window's points, of target pixels at most (0: any) */
static int window_parts(double wt, double target)
{
    return target > 0.0 ? (int)std::min(64.0, std::max(1.0, ceil(wt / target))) : 1;
}

/* The items of one block's windows. */
static void block_windows(const hl_handle *h, const plan_img &im, int img, int sl, int cap,
                          double target, std::vector<plan_region> &reg)
{
    const plan_band p = block_band(h, im.w, im.h, sl);
    const int tx = (im.w + HL_TILE_W - 1) / HL_TILE_W, ty = (im.h + HL_TILE_H - 1) / HL_TILE_H;
    int rows;
    const int n = band_windows(p, cap, &rows);
    for (int j = 0; j < n; j++) {
        plan_region r;
        memset(&r.it, 0, sizeof(r.it));
        r.it.img = img;
        r.it.slice = sl;
        r.it.tx = tx << 16;
        r.it.ty = ty << 16;
        r.it.slab = -1;
        r.it.win = 1;
        r.it.nseg = (ty + HL_VOTE_RUNS / 2 - 1) / (HL_VOTE_RUNS / 2);
        r.it.adv = rows;
        r.it.off0 = p.first + j * rows;
        r.it.lo = (float)(r.it.off0 * h->p.derho - p.out);
        r.it.hi = (float)((r.it.off0 + rows) * h->p.derho + p.out);
        r.it.tang = (float)p.tang;
        r.blk = img * (h->Tp / HL_SLICE) + sl;
        r.wt = window_weight(h, p, (double)im.w * im.h, j, rows);
        r.it.nparts = window_parts(r.wt, target);
        r.wt /= r.it.nparts;
        for (r.it.part = 0; r.it.part < r.it.nparts; r.it.part++)
            reg.push_back(r);
    }
}

static bool heavier(const plan_region &a, const plan_region &c) { return a.wt > c.wt; }

/* A list schedule of the items, heaviest first: when each starts; the end. */
static double plan_schedule(std::vector<plan_region> &reg, int ctas, std::vector<double> &start)
{
    std::stable_sort(reg.begin(), reg.end(), heavier);
    std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
    double makespan = 0.0;
    start.resize(reg.size());
    for (size_t i = 0; i < reg.size(); i++) {
        start[i] = 0.0;
        if ((int)i >= std::max(ctas, 1)) {
            start[i] = free_at.top();
            free_at.pop();
        }
        makespan = std::max(makespan, start[i] + reg[i].wt);
        free_at.push(start[i] + reg[i].wt);
    }
    return makespan;
}

/* The plan of regions: whole images where they fit a window or can slide and weigh
 * no more than a CTA's share, else grids of regions (windows where not even a tile's
 * rows fit one). */
static void plan_regions(const hl_handle *h, const plan_img *im, int n, int cap, int ctas,
                           const std::vector<slice_ext> &ext, double total,
                           std::vector<plan_region> &reg)
{
    const int slices = h->Tp / HL_SLICE;
    const double wcap = std::max(total / (HL_PLAN_SHARE * std::max(ctas, 1)), HL_MIN_REGION);
    /* A block heavier than that is one item all the same, one such a CTA, if it is
     * no more than a CTA's share: the rest, split, fill what is left.  A whole block
     * needs no slabs: 21 images of 2048 x 2048, T = 360, voted 271 and merged 18 us
     * instead of 278 and 50 with every block in two or more regions. */
    const double share = total / std::max(ctas, 1);
    int big = 0;
    for (int i = 0; i < n; i++) {
        const int w = im[i].w, hh = im[i].h;
        const int tx = (w + HL_TILE_W - 1) / HL_TILE_W, ty = (hh + HL_TILE_H - 1) / HL_TILE_H;
        for (int sl = 0; sl < slices; sl++) {
            double n_min = std::max(1.0, ceil((double)w * hh / wcap));
            hl_vote_item whole;
            if (n_min > 1.0 && big < ctas &&
                (double)w * hh + HL_ROW_PIXELS * region_rows(ext[sl], w, hh) <= share &&
                (region_rows(ext[sl], w, hh) <= cap ||
                 slide_item(h, ext[sl], w, hh, sl, cap, &whole))) {
                n_min = 1.0;
                big++;
            }
            if (n_min <= 1.0 && slide_item(h, ext[sl], w, hh, sl, cap, &whole)) {
                whole.img = i;
                plan_region r;
                r.it = whole;
                r.blk = i * slices + sl;
                r.wt = (double)w * hh + HL_ROW_PIXELS * region_rows(ext[sl], w, hh);
                reg.push_back(r);
                continue;
            }
            int nx, ny;
            if (!best_grid(ext[sl], w, hh, cap, n_min, &nx, &ny)) {
                block_windows(h, im[i], i, sl, cap, 0.0, reg);
                continue;
            }
            for (int y = 0; y < ny; y++)
                for (int x = 0; x < nx; x++) {
                    const int x0 = tx * x / nx, x1 = tx * (x + 1) / nx;
                    const int y0 = ty * y / ny, y1 = ty * (y + 1) / ny;
                    const double gw = std::min(x1 * HL_TILE_W, w) - x0 * HL_TILE_W;
                    const double gh = std::min(y1 * HL_TILE_H, hh) - y0 * HL_TILE_H;
                    plan_region r;
                    memset(&r.it, 0, sizeof(r.it));
                    r.it.img = i;
                    r.it.slice = sl;
                    r.it.tx = x0 | ((x1 - x0) << 16);
                    r.it.ty = y0 | ((y1 - y0) << 16);
                    r.it.nseg = 1;
                    r.blk = i * slices + sl;
                    /* a region that the slice's rho 0 crosses votes by the
                     * sign of each vote, about 1.4 times the time */
                    const int k0 = sl * HL_SLICE, k1 = std::min(k0 + HL_SLICE, h->T) - 1;
                    const bool mixed = h->h_cos[k1] < 0.0f &&
                                       (x0 * h->h_cos[k0] * HL_TILE_W +
                                            y1 * h->h_sin[k0] * HL_TILE_H > 0.0f) &&
                                       (x1 * h->h_cos[k1] * HL_TILE_W +
                                            y0 * h->h_sin[k1] * HL_TILE_H < 0.0f);
                    r.wt = gw * gh * (mixed ? 1.4 : 1.0) +
                           HL_ROW_PIXELS * region_rows(ext[sl], gw, gh);
                    reg.push_back(r);
                }
        }
    }
    /* the late starters of a list schedule, halved along their longer side */
    std::vector<double> start;
    double makespan = plan_schedule(reg, ctas, start);
    const size_t n0 = reg.size();
    for (size_t i = 0; i < n0; i++) {
        plan_region r = reg[i];
        if (!(start[i] > 0.6 * makespan && r.wt > 0.25 * wcap && r.wt >= 2.0 * HL_MIN_REGION &&
              !r.it.win && r.it.nseg == 1))
            continue;
        const int txn = r.it.tx >> 16, tyn = r.it.ty >> 16;
        plan_region a = r, b = r;
        if (txn * HL_TILE_W >= tyn * HL_TILE_H && txn > 1 && tyn <= HL_VOTE_RUNS) {
            const int x0 = r.it.tx & 0xffff, m = txn / 2;
            a.it.tx = x0 | (m << 16);
            b.it.tx = (x0 + m) | ((txn - m) << 16);
        } else if (tyn > 1) {
            const int y0 = r.it.ty & 0xffff, m = tyn / 2;
            a.it.ty = y0 | (m << 16);
            b.it.ty = (y0 + m) | ((tyn - m) << 16);
        } else {
            continue;
        }
        a.wt = b.wt = 0.6 * r.wt;
        reg[i] = a;
        reg.push_back(b);
    }
    std::stable_sort(reg.begin(), reg.end(), heavier);
}

/* The plan of windows of at most cap rows, blocks that fit one whole. */
static void plan_in_windows(const hl_handle *h, const plan_img *im, int n, int cap, double target,
                            const std::vector<slice_ext> &ext, std::vector<plan_region> &reg)
{
    const int slices = h->Tp / HL_SLICE;
    for (int i = 0; i < n; i++)
        for (int sl = 0; sl < slices; sl++) {
            const double rows = region_rows(ext[sl], im[i].w, im[i].h);
            if (rows > cap) {
                block_windows(h, im[i], i, sl, cap, target, reg);
                continue;
            }
            plan_region r;
            memset(&r.it, 0, sizeof(r.it));
            r.it.img = i;
            r.it.slice = sl;
            r.it.tx = ((im[i].w + HL_TILE_W - 1) / HL_TILE_W) << 16;
            r.it.ty = ((im[i].h + HL_TILE_H - 1) / HL_TILE_H) << 16;
            r.it.nseg = 1;
            r.blk = i * slices + sl;
            r.wt = (double)im[i].w * im[i].h + HL_ROW_PIXELS * rows;
            reg.push_back(r);
        }
    std::stable_sort(reg.begin(), reg.end(), heavier);
}

/* Pixels that a launch of items of these weights takes: its heaviest item, a CTA's
 * share (items do not share out evenly) or, in a list schedule of a little more items
 * than CTAs, the first two on one CTA; and the slabs' rows. */
static double plan_length(std::vector<double> &wt, double sum, double most, double slab_rows,
                          int ctas)
{
    ctas = std::max(ctas, 1);
    double len = std::max(1.1 * (sum + HL_ITEM_PIXELS * (double)wt.size()) / ctas,
                          most + HL_ITEM_PIXELS);
    if ((int)wt.size() > ctas) {
        std::nth_element(wt.begin(), wt.begin() + ctas, wt.end(), std::greater<double>());
        len = std::max(len, 2.0 * (wt[(size_t)ctas] + HL_ITEM_PIXELS));
    }
    return len + (slab_rows > 0.0 ? HL_MERGE_PIXELS : 0.0) + slab_rows * HL_SLAB_PIXELS / ctas;
}

/* Is a plan of windows the shorter one?  *cap: the windows' rows at most, in and out;
 * *target: pixels of a part at most, 0 for whole windows. */
static bool windows_win(const hl_handle *h, const plan_img *im, int n, int ctas,
                        const std::vector<slice_ext> &ext, double total, int *cap, double *target)
{
    const int slices = h->Tp / HL_SLICE;
    const double wcap = std::max(total / (HL_PLAN_SHARE * std::max(ctas, 1)), HL_MIN_REGION);
    double sum = 0.0, most = 0.0, slab_rows = 0.0, best = 1e300;
    bool grid = true, win = false;
    std::vector<double> wt, part;
    for (int i = 0; i < n && grid; i++)
        for (int sl = 0; sl < slices && grid; sl++) {
            const double area = (double)im[i].w * im[i].h;
            int nx = 1, ny = 1;
            hl_vote_item it;
            if (!(area <= wcap && slide_item(h, ext[sl], im[i].w, im[i].h, sl, *cap, &it)))
                grid = best_grid(ext[sl], im[i].w, im[i].h, *cap,
                                 std::max(1.0, ceil(area / wcap)), &nx, &ny);
            const double rows = region_rows(ext[sl], (double)im[i].w / nx, (double)im[i].h / ny);
            const double w = area / (nx * ny) + HL_ROW_PIXELS * rows;
            wt.insert(wt.end(), (size_t)nx * ny, w);
            sum += nx * ny * w;
            most = std::max(most, w);
            slab_rows += nx * ny > 1 ? nx * ny * rows : 0.0;
        }
    if (grid)
        best = plan_length(wt, sum, most, slab_rows, ctas);
    std::vector<plan_band> band;
    for (int i = 0; i < n; i++)
        for (int sl = 0; sl < slices; sl++)
            band.push_back(block_band(h, im[i].w, im[i].h, sl));
    for (int c = *cap, top = *cap, worse = 0; c >= 128 && worse < 2; c = c * 2 / 3) {
        wt.clear();
        sum = most = 0.0;
        for (int i = 0; i < n; i++)
            for (int sl = 0; sl < slices; sl++) {
                const plan_band &b = band[(size_t)(i * slices + sl)];
                const double area = (double)im[i].w * im[i].h;
                const double whole = region_rows(ext[sl], im[i].w, im[i].h);
                int rows = 0;
                const int nw = whole > c ? band_windows(b, c, &rows) : 1;
                for (int j = 0; j < nw; j++) {
                    wt.push_back(rows ? window_weight(h, b, area, j, rows)
                                      : area + HL_ROW_PIXELS * whole);
                    sum += wt.back();
                    most = std::max(most, wt.back());
                }
            }
        /* whole, then in parts: every item of a block that has any goes through slabs */
        const double share = std::max(sum / std::max(ctas, 1), 0.5 * HL_MIN_REGION);
        bool better = false;
        for (double f : {0.0, 2.0, 1.5, 1.0}) {
            if (f > 0.0 && most <= f * share)
                continue;
            part.clear();
            slab_rows = 0.0;
            double heaviest = 0.0;
            size_t at = 0;
            for (int i = 0; i < n; i++)
                for (int sl = 0; sl < slices; sl++) {
                    const double whole = region_rows(ext[sl], im[i].w, im[i].h);
                    /* a slab's groups of eight columns are as tall as these lie apart */
                    const double apart = 0.5 * sqrt((double)im[i].w * im[i].w +
                                                    (double)im[i].h * im[i].h) *
                                         std::min(7.0 * h->p.detheta, 1.0) / h->p.derho;
                    int rows = 0;
                    const int nw =
                        whole > c ? band_windows(band[(size_t)(i * slices + sl)], c, &rows) : 1;
                    const size_t before = part.size();
                    for (int j = 0; j < nw; j++, at++) {
                        const int np = rows ? window_parts(wt[at], f * share) : 1;
                        part.insert(part.end(), (size_t)np, wt[at] / np);
                        heaviest = std::max(heaviest, wt[at] / np);
                    }
                    const size_t items = part.size() - before;
                    slab_rows += items > (size_t)nw ? (double)items * (rows + apart) : 0.0;
                }
            const double len = plan_length(part, sum, heaviest, slab_rows, ctas);
            if (len < best) {
                best = len;
                *cap = c;
                *target = f * share;
                win = better = true;
            }
        }
        worse = better || c == top ? 0 : worse + 1;
        if (n * slices >= 2 * ctas)
            break;   /* items enough: smaller windows only repeat votes */
    }
    return win;
}

/* Plans the vote of n images with windows of at most cap rows on ctas
 * persistent CTAs; slabs: there is memory for them. */
static int make_plan(const hl_handle *h, const plan_img *im, int n, int cap, int ctas,
                     bool slabs, vote_plan *pl)
try {
    const int slices = h->Tp / HL_SLICE;
    std::vector<slice_ext> ext;
    slice_extents(h, ext);
    double total = 0.0;
    pl->exact = 0;
    pl->add = !slabs;
    pl->part16 = 1;
    for (int i = 0; i < n; i++) {
        if (im[i].R >= (1 << 22))
            pl->exact = 1;
        for (int sl = 0; sl < slices; sl++)
            total += (double)im[i].w * im[i].h +
                     HL_ROW_PIXELS * std::min(region_rows(ext[sl], im[i].w, im[i].h), 4.0 * cap);
    }
    std::vector<plan_region> reg;
    int wcap = cap;
    double target = 0.0;
    const bool small = n * slices < 2 * ctas && total / std::max(ctas, 1) < HL_SMALL_PIXELS;
    if ((h->p.derho < 1.0 || small) &&
        windows_win(h, im, n, ctas, ext, total, &wcap, &target))
        plan_in_windows(h, im, n, wcap, target, ext, reg);
    else
        plan_regions(h, im, n, cap, ctas, ext, total, reg);
    bool slides = false;
    int win_rows = 0;
    for (const plan_region &r : reg) {
        slides |= !r.it.win && r.it.nseg > 1;
        win_rows = std::max(win_rows, r.it.win ? r.it.adv : 0);
    }
    pl->win = win_rows > 0;
    /* slabs and merge blocks of the blocks with several items */
    std::vector<int> count((size_t)n * slices, 0), first((size_t)n * slices, 0);
    std::vector<int> at((size_t)n * slices, -1);   /* in pl->blocks */
    std::vector<char> parts((size_t)n * slices, 0);
    for (const plan_region &r : reg)
        parts[(size_t)r.blk] |= r.it.nparts > 1;
    for (const plan_region &r : reg)   /* whole windows are final */
        if (!r.it.win || parts[(size_t)r.blk])
            count[(size_t)r.blk]++;
    pl->blocks.clear();
    int nslab = 0;
    for (int b = 0; b < n * slices; b++)
        if (count[(size_t)b] > 1) {
            first[(size_t)b] = nslab;
            at[(size_t)b] = (int)pl->blocks.size();
            pl->blocks.push_back({b / slices, b % slices, nslab, count[(size_t)b], 0x7fffffff, 0});
            nslab += count[(size_t)b];
        }
    pl->slabs.assign((size_t)nslab, hl_slab{});
    for (const plan_region &r : reg) {
        if (r.it.win && !parts[(size_t)r.blk])
            continue;
        const int w = im[r.it.img].w, hh = im[r.it.img].h;
        pl->part16 &= hl_part16_ok(h->p.derho, std::min((r.it.tx >> 16) * HL_TILE_W, w),
                                   std::min((r.it.ty >> 16) * HL_TILE_H, hh));
    }
    pl->items.resize(reg.size());
    pl->scratch_units = 0;
    long long max_scratch = 0;
    for (int i = 0; i < n; i++)
        max_scratch += 8LL * im[i].R * h->Tp;
    /* slabs are numbered in 31 bits */
    max_scratch = std::min(std::max(max_scratch, HL_MAX_SCRATCH), 64LL * 0x7fffffff);
    double most = std::max(8, win_rows);
    std::vector<double> bend((size_t)slices * 4);
    for (size_t g = 0; g < bend.size(); g++)
        bend[g] = slab_bend(h, (int)g * 8);
    for (size_t i = 0; i < reg.size(); i++) {
        hl_vote_item it = reg[i].it;
        const int w = im[it.img].w, hh = im[it.img].h;
        const int x1 = std::min(((it.tx & 0xffff) + (it.tx >> 16)) * HL_TILE_W, w);
        const int y1 = std::min(((it.ty & 0xffff) + (it.ty >> 16)) * HL_TILE_H, hh);
        const double rows = region_rows(ext[it.slice], x1 - (it.tx & 0xffff) * HL_TILE_W,
                                        y1 - (it.ty & 0xffff) * HL_TILE_H);
        if (!it.win)
            most = std::max(most, std::min(rows, (double)cap));
        const size_t b = (size_t)reg[i].blk;
        it.slab = -1;
        if (count[b] > 1) {
            hl_slab sl = {};
            if (it.win)
                window_groups(h, im[it.img], it, &sl);
            else
                slab_groups(h, im[it.img], it, x1, y1, &bend[(size_t)it.slice * 4], &sl);
            long long units = 0;
            for (int g = 0; g < 4; g++) {
                sl.o[g] = (int)units;
                units += sl.n[g];
                it.gb[g] = sl.b[g];
                it.gn[g] = sl.n[g];
                it.go[g] = sl.o[g];
            }
            pl->add |= pl->scratch_units + units > max_scratch / (pl->part16 ? 64 : 128);
            if (!pl->add) {
                it.slab = sl.at = (int)pl->scratch_units;
                pl->scratch_units += units;
                hl_merge_block &mb = pl->blocks[(size_t)at[b]];
                mb.lo = std::min(mb.lo, sl.lo);
                mb.hi = std::max(mb.hi, sl.hi);
                pl->slabs[(size_t)first[b]++] = sl;
            }
        }
        pl->items[i] = it;
    }
    if (pl->add) {
        for (hl_vote_item &it : pl->items)
            it.slab = -1;
        pl->blocks.clear();
        pl->slabs.clear();
        pl->scratch_units = 0;
    }
    pl->chunks = 1;
    for (const hl_merge_block &mb : pl->blocks)
        pl->chunks = std::max(pl->chunks, (unsigned)(mb.hi - mb.lo + 15) / 16);
    pl->win_rows = slides ? cap : std::min(cap, ((int)most + 7) / 8 * 8);
    return HL_NO_ERROR;
} catch (const std::bad_alloc &) {   /* many windows of a very fine step */
    return HL_OUT_OF_MEM;
}

/* rows a window may have: the override (at least what one tile needs at a
 * whole rho step) or what fits next to the staging ring */
static int plan_cap(const hl_handle *h)
{
    const int maxr = hl_vote_max_rows();
    if (h->win_rows_override <= 0)
        return maxr;
    return std::min(maxr, std::max(h->win_rows_override, 168));
}
static int vote_threads(const hl_handle *h)
{
    return h->threads_override > 0 ? h->threads_override : 1024;
}
/* persistent CTAs an SM holds with windows of `rows` rows */
static int vote_ctas(const hl_handle *h, int rows, int threads)
{
    const size_t smem = hl_vote_smem_bytes(rows);
    const int per_sm = std::max(1, std::min(2048 / threads, (int)((228u * 1024u) / (smem + 1024))));
    return std::max(h->sms, 1) * per_sm;
}

static size_t plan_bytes(const vote_plan &p)
{
    return p.items.size() * sizeof(hl_vote_item) + p.blocks.size() * sizeof(hl_merge_block) +
           p.slabs.size() * sizeof(hl_slab);
}
/* slabs (read in 16-byte pieces), items, blocks */
static void plan_copy(const vote_plan &p, unsigned char *dst)
{
    size_t o = 0;
    const auto put = [&](const void *src, size_t n) {
        if (n)
            memcpy(dst + o, src, n);
        o += n;
    };
    put(p.slabs.data(), p.slabs.size() * sizeof(hl_slab));
    put(p.items.data(), p.items.size() * sizeof(hl_vote_item));
    put(p.blocks.data(), p.blocks.size() * sizeof(hl_merge_block));
}
static void plan_args(const vote_plan &p, const unsigned char *d_plan, unsigned char *scratch,
                      hl_vote_args *va, hl_merge_args *ma)
{
    size_t o = p.slabs.size() * sizeof(hl_slab);
    ma->slabs = reinterpret_cast<const hl_slab *>(d_plan);
    va->items = reinterpret_cast<const hl_vote_item *>(d_plan + o);
    va->nitems = (int)p.items.size();
    va->win = p.win;
    va->win_rows = p.win_rows;
    va->exact = p.exact;
    va->part16 = p.part16;
    va->add = p.add;
    va->scratch = scratch;
    o += p.items.size() * sizeof(hl_vote_item);
    ma->imgs = va->imgs;
    ma->img0 = va->img0;
    ma->T = va->T;
    ma->Tp = va->Tp;
    ma->scratch = scratch;
    ma->blocks = reinterpret_cast<const hl_merge_block *>(d_plan + o);
    ma->nblocks = (int)p.blocks.size();
    ma->chunks = p.chunks;
    ma->part16 = p.part16;
    ma->cand = va->cand;
}

/* Uploads the handle's plan on s, behind whatever there still reads the previous
 * one; the staging copy is rewritten once the previous upload has read it.  A
 * stream under capture is refused: a replay would read the staging copy as later
 * calls leave it. */
static int plan_upload(hl_handle *h, cudaStream_t s)
{
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CK(cudaStreamIsCapturing(s, &cap));
    if (cap != cudaStreamCaptureStatusNone)
        return HL_CUDA_ERROR;
    const size_t bytes = plan_bytes(*h->plan);
    if (!h->plan_event) {
        CK(cudaEventCreateWithFlags(&h->plan_read, cudaEventDisableTiming));
        h->plan_event = 1;
    }
    CK(cudaEventSynchronize(h->plan_read));
    int rc;
    if ((rc = grow_host(&h->h_plan, &h->cap_hplan, bytes)) != HL_NO_ERROR ||
        (rc = grow((void **)&h->d_plan, &h->cap_plan, bytes)) != HL_NO_ERROR)
        return rc;
    plan_copy(*h->plan, h->h_plan);
    CK(cudaMemcpyAsync(h->d_plan, h->h_plan, bytes, cudaMemcpyHostToDevice, s));
    CK(cudaEventRecord(h->plan_read, s));
    return HL_NO_ERROR;
}

/* The handle's plan for a w x hh ROI, uploaded, and room for its slabs and noted
 * candidates. */
static int handle_plan(hl_handle *h, int w, int hh, int R, int rho_min, cudaStream_t s)
{
    const int cap = plan_cap(h), threads = vote_threads(h);
    if (!(h->plan && h->plan_w == w && h->plan_h == hh && h->plan_R == R && h->plan_T == h->T &&
          h->plan_derho == h->p.derho && h->plan_detheta == h->p.detheta && h->plan_cap == cap &&
          h->plan_thr == threads)) {
        if (!h->plan && !(h->plan = new (std::nothrow) vote_plan()))
            return HL_OUT_OF_MEM;
        h->plan_w = 0;   /* not valid until the upload below */
        if (h->acc_state == ACC_UNREACHED)
            h->acc_state = ACC_ANY;
        const plan_img im = {w, hh, R, rho_min};
        int rc = make_plan(h, &im, 1, cap, std::max(h->sms, 1), true, h->plan);
        if (rc != HL_NO_ERROR)
            return rc;
        if ((rc = plan_upload(h, s)) != HL_NO_ERROR)
            return rc;
        h->plan_w = w;
        h->plan_h = hh;
        h->plan_R = R;
        h->plan_T = h->T;
        h->plan_derho = h->p.derho;
        h->plan_detheta = h->p.detheta;
        h->plan_cap = cap;
        h->plan_thr = threads;
    }
    int rc = grow((void **)&h->d_scratch, &h->cap_scratch, plan_scratch(*h->plan));
    if (rc == HL_OUT_OF_MEM && !h->plan->add) {
        /* no room for the slabs: the form without them */
        const plan_img im = {w, hh, R, rho_min};
        h->plan_w = 0;
        if ((rc = make_plan(h, &im, 1, cap, std::max(h->sms, 1), false, h->plan)) != HL_NO_ERROR ||
            (rc = plan_upload(h, s)) != HL_NO_ERROR)
            return rc;
        h->plan_w = w;
        rc = grow((void **)&h->d_scratch, &h->cap_scratch, plan_scratch(*h->plan));
    }
    if (rc != HL_NO_ERROR)
        return rc;
    return grow((void **)&h->d_cand, &h->cap_cand,
                sizeof(unsigned long long) * (65536 + (size_t)R * h->Tp / 128));
}

/* New buffers are cleared on the call's stream: the default stream's order does not
 * reach a non-blocking one. */
static int ensure_image(hl_handle *h, const hl_geom &g, int w, int hh, cudaStream_t s)
{
    int rc;
    size_t ntiles = (size_t)g.tiles_x * g.tiles_y;
    if ((rc = grow((void **)&h->d_pts, &h->cap_pts,
                   sizeof(float2) * ((size_t)w * hh + 16))) != HL_NO_ERROR)
        return rc;
    if (h->cap_tiles < ntiles + 1 || !h->d_tile_state || !h->d_tile_off) {
        size_t cap = 0;
        if ((rc = grow((void **)&h->d_tile_state, &cap,
                       sizeof(unsigned long long) * (ntiles + 1))) != HL_NO_ERROR)
            return rc;
        CK(cudaMemsetAsync(h->d_tile_state, 0, cap, s));
        size_t cap2 = 0;
        if ((rc = grow((void **)&h->d_tile_off, &cap2,
                       sizeof(int) * (ntiles + 1))) != HL_NO_ERROR)
            return rc;
        h->cap_tiles = std::min(cap / sizeof(unsigned long long),
                                cap2 / sizeof(int));
    }
    return HL_NO_ERROR;
}

/* Peak candidates: the list and its room; a threshold that only
 * peaks-to-be clear leaves a few hundred per image, and past the room the
 * peak pass scans the accumulators instead.  A null list: no noting. */
static hl_cand_list cand_list(unsigned long long *e, size_t cap_bytes, int *count)
{
    hl_cand_list c;
    c.e = e;
    c.count = count;
    c.cap = (int)std::min(cap_bytes / sizeof(unsigned long long), (size_t)0x7fffffff);
    c.pad = 0;
    return c;
}

static int ensure_acc(hl_handle *h, int R, int linesmax)
{
    int rc;
    size_t bins = (size_t)R * h->Tp;
    if (h->cap_acc < sizeof(int32_t) * bins)
        h->acc_state = ACC_ANY;   /* another buffer, also after a failed allocation */
    if ((rc = grow((void **)&h->d_acc, &h->cap_acc, sizeof(int32_t) * bins)) !=
        HL_NO_ERROR)
        return rc;
    /* peaks never sit next to each other along theta: at most ceil(T/2)
     * per rho row */
    size_t maxpk = (size_t)R * ((h->T + 1) / 2) + 32;
    if ((rc = grow((void **)&h->d_keys, &h->cap_keys,
                   sizeof(unsigned long long) * maxpk)) != HL_NO_ERROR)
        return rc;
    size_t lm = (size_t)std::max(linesmax, 1);
    size_t rbytes = sizeof(hl_result_hdr) + sizeof(hl_line) * lm;
    if (h->cap_result < rbytes || !h->d_result) {
        if ((rc = grow((void **)&h->d_result, &h->cap_result, rbytes)) !=
            HL_NO_ERROR)
            return rc;
        if (h->h_result)
            cudaFreeHost(h->h_result);
        h->h_result = nullptr;
        CK(cudaMallocHost(&h->h_result, h->cap_result));
    }
    return HL_NO_ERROR;
}

static int key_cap(const hl_handle *h)
{
    size_t c = h->cap_keys / sizeof(unsigned long long);
    return (int)std::min(c, (size_t)0x7fffffff);
}

static int roi_of(const hl_image_desc *img, hl_roi *roi)
{
    if (!img || !img->data)
        return HL_NULL_POINTER;
    /* okano_3_0/Image.h:218-258: the ROI must lie inside the image */
    if (img->width <= 0 || img->height <= 0 || img->pitch < (size_t)img->width)
        return HL_INVALID_DATA;
    if (img->roi_x1 < 0 || img->roi_y1 < 0 || img->roi_x2 > img->width ||
        img->roi_y2 > img->height || img->roi_x2 <= img->roi_x1 ||
        img->roi_y2 <= img->roi_y1)
        return HL_INVALID_DATA;
    roi->w = img->roi_x2 - img->roi_x1;
    roi->h = img->roi_y2 - img->roi_y1;
    if (roi->w > HL_MAX_SIDE || roi->h > HL_MAX_SIDE)
        return HL_INVALID_DATA;
    roi->base = img->data + (size_t)img->roi_y1 * img->pitch + img->roi_x1;
    roi->pitch = (long)img->pitch;
    return HL_NO_ERROR;
}

/* hl_launch_compact on a ticket counter of its own (the number of tickets a
 * launch takes is not known) */
static cudaError_t launch_compact_groups(hl_handle *h, hl_compact_args *ca, cudaStream_t s)
{
    const cudaError_t e = cudaMemsetAsync(h->d_counters + 12, 0, sizeof(unsigned), s);
    if (e != cudaSuccess)
        return e;
    ca->ticket = reinterpret_cast<unsigned *>(h->d_counters + 12);
    ca->ticket_base = 0;
    return hl_launch_compact(ca, s);
}

/* Stage (a) of one image's ROI into h->d_pts (float2, tile-major, odd tiles
 * padded), h->d_tile_off and the point count h->d_counters[2]: about one
 * CTA per SM when they fit at once, else one CTA per 4-tile group. */
static int launch_compaction(hl_handle *h, const hl_roi &roi, const hl_geom &g,
                             cudaStream_t s)
{
    const int ntiles = g.tiles_x * g.tiles_y;
    hl_compact_args ca;
    memset(&ca, 0, sizeof(ca));
    ca.roi = roi;
    ca.tiles_x = g.tiles_x;
    ca.ntiles = ntiles;
    ca.tile_state = h->d_tile_state;
    ca.ticket = reinterpret_cast<unsigned *>(h->d_counters + 3);
    ca.ticket_base = h->ticket_base;
    if (++h->epoch >= (1u << 30)) {
        CK(cudaMemsetAsync(h->d_tile_state, 0,
                           sizeof(unsigned long long) * h->cap_tiles, s));
        h->epoch = 1;
    }
    ca.epoch = h->epoch;
    ca.pts = nullptr;
    ca.pts_f2 = reinterpret_cast<float2 *>(h->d_pts);
    ca.tile_off = h->d_tile_off;
    ca.count = h->d_counters + 2;
    ca.status = h->d_counters + 1;
    const int nct = hl_compact_persist_ctas(ntiles, h->sms);
    if (nct > 0) {
        CK(hl_launch_compact_persist(&ca, nct, s));
        h->ticket_base += (unsigned)nct;
    } else {
        CK(launch_compact_groups(h, &ca, s));
    }
    return HL_NO_ERROR;
}

/* stages (a) + (b) into h->d_acc ([R][Tp]) */
static int run_ab(hl_handle *h, const hl_roi &roi, const hl_geom &g, bool peaks,
                  cudaStream_t s, int *launches)
{
    const int ntiles = g.tiles_x * g.tiles_y;

    hl_vote_args va;
    memset(&va, 0, sizeof(va));
    va.imgs = nullptr;
    va.img0.pts = reinterpret_cast<const float2 *>(h->d_pts);
    va.img0.tile_off = h->d_tile_off;
    va.img0.ntiles = ntiles;
    va.img0.tiles_x = g.tiles_x;
    va.img0.w = roi.w;
    va.img0.h = roi.h;
    va.img0.rho_min = g.rho_min;
    va.img0.R = g.numrho;
    va.img0.threshold = h->p.threshold;
    va.img0.acc = h->d_acc;
    va.cosv = h->d_cos;
    va.sinv = h->d_sin;
    va.T = h->T;
    va.Tp = h->Tp;
    va.irho = (float)(1.0 / h->p.derho);   /* okano_3_0/HoughLine.cu:107 */
    va.status = h->d_counters + 1;
    int rc = handle_plan(h, roi.w, roi.h, g.numrho, g.rho_min, s);
    if (rc != HL_NO_ERROR)
        return rc;
    /* bins above the threshold are noted where their final count is known;
     * the accumulator entry points take no peaks */
    va.cand = peaks && !h->plan->add
                  ? cand_list(h->d_cand, h->cap_cand, h->d_counters + 10 + h->cand_par)
                  : cand_list(nullptr, 0, nullptr);
    hl_merge_args ma;
    memset(&ma, 0, sizeof(ma));
    plan_args(*h->plan, h->d_plan, h->d_scratch, &va, &ma);
    const int threads = vote_threads(h);
    const int ctas = vote_ctas(h, va.win_rows, threads);
    if (va.add)
        h->acc_state = ACC_ANY;
    if (h->acc_state == ACC_ANY || (peaks && h->acc_state != ACC_ZERO)) {
        CK(cudaMemsetAsync(h->d_acc, 0, h->cap_acc, s));
        CK(cudaMemsetAsync(h->d_counters + 10, 0, 2 * sizeof(int), s));
    }
    /* with peaks the tail clears what is stored (set when it is launched) */
    h->acc_state = peaks || va.add ? ACC_ANY : ACC_UNREACHED;

    prof_mark(h, 0, s);
    rc = launch_compaction(h, roi, g, s);
    if (rc != HL_NO_ERROR)
        return rc;
    (*launches)++;
    prof_mark(h, 1, s);

    const int grid = std::min(va.nitems, ctas);
    va.work = reinterpret_cast<unsigned *>(h->d_counters + 9);
    va.work_base = h->work_base;
    CK(hl_launch_vote(&va, threads, grid, s));
    /* every CTA takes one ticket per item plus one that finds no item */
    h->work_base += (unsigned)(va.nitems + grid);
    (*launches)++;
    if (ma.nblocks > 0) {
        CK(hl_launch_merge(&ma, s));
        (*launches)++;
    }
    prof_mark(h, 2, s);
    return HL_NO_ERROR;
}

/* stage (c) over h->d_acc */
/* the tail's arguments for one image: the handle's keys and counters, the
 * result records into lines_dev (or the handle's result buffer) */
static void final_args(hl_handle *h, const hl_geom &g, int linesmax, hl_line *lines_dev,
                       int *count_dev, hl_final_args *fa)
{
    memset(fa, 0, sizeof(*fa));
    fa->imgs = nullptr;
    fa->img0.keys = h->d_keys;
    fa->img0.ncand = h->d_counters + 0;
    fa->img0.cap = key_cap(h);
    fa->img0.rho_min = g.rho_min;
    fa->img0.ref_numrho = g.ref_numrho;
    fa->img0.pad = 0;
    fa->T = h->T;
    fa->detheta = h->p.detheta;
    fa->thresdis = h->p.thresdis;
    fa->thresang = h->p.thresang;
    fa->linesmax = linesmax;
    fa->hdr = reinterpret_cast<hl_result_hdr *>(h->d_result);
    fa->img0.lines = lines_dev ? lines_dev
                               : reinterpret_cast<hl_line *>(h->d_result +
                                                             sizeof(hl_result_hdr));
    fa->status = h->d_counters + 1;
    fa->img0.count_out = count_dev;
}

/* noted: the vote noted the peak candidates (d_cand) */
static int run_c(hl_handle *h, const hl_geom &g, bool noted, int linesmax,
                 hl_line *lines_dev, int *count_dev, cudaStream_t s,
                 int *launches)
{
    hl_peak_args pa;
    pa.imgs = nullptr;
    pa.img0.acc = h->d_acc;
    pa.img0.keys = h->d_keys;
    pa.img0.ncand = h->d_counters + 0;
    pa.img0.R = g.numrho;
    pa.img0.cap = key_cap(h);
    pa.img0.threshold = h->p.threshold;
    pa.img0.pad = 0;
    pa.chunks = nullptr;
    /* units of HL_PEAK_FLAT int4; the kernel indexes the accumulator's int4
     * in 32 bits */
    if ((long long)g.numrho * (h->Tp / 4) >= (1LL << 32))
        return HL_OP_OVERFLOW;
    pa.nchunks = (int)(((long long)g.numrho * (h->Tp / 4) + HL_PEAK_FLAT - 1) / HL_PEAK_FLAT);
    pa.T = h->T;
    pa.Tp = h->Tp;
    pa.status = h->d_counters + 1;
    pa.cand = noted ? cand_list(h->d_cand, h->cap_cand, h->d_counters + 10 + h->cand_par)
                    : cand_list(nullptr, 0, nullptr);
    CK(hl_launch_peaks(&pa, s));
    (*launches)++;
    prof_mark(h, 3, s);

    hl_final_args fa;
    final_args(h, g, linesmax, lines_dev, count_dev, &fa);
    if (noted) {
        fa.clear = pa.cand;
        fa.acc = h->d_acc;
        fa.acc_ints = (long long)g.numrho * h->Tp;
        fa.Tp = h->Tp;
        fa.cand_count = h->d_counters + 10 + (h->cand_par ^ 1);
    }
    CK(hl_launch_finalize(&fa, 1, s));
    if (noted) {
        h->cand_par ^= 1;
        h->acc_state = ACC_ZERO;
    }
    (*launches)++;
    prof_mark(h, 4, s);
    return HL_NO_ERROR;
}

/* After a device-side failure the ticket / work counters may not have
 * advanced by what the host expects: zero them and their bases. */
static void reset_counters(hl_handle *h, cudaStream_t s)
{
    cudaMemsetAsync(h->d_counters, 0, 16 * sizeof(int), s);
    cudaStreamSynchronize(s);
    h->ticket_base = 0;
    h->work_base = 0;
    h->acc_state = ACC_ANY;
}

static int fetch_result(hl_handle *h, int *linesmax, hl_line *lines,
                        cudaStream_t s)
{
    int lm = std::max(*linesmax, 0);
    size_t bytes = sizeof(hl_result_hdr) + sizeof(hl_line) * (size_t)lm;
    CK(cudaMemcpyAsync(h->h_result, h->d_result, bytes, cudaMemcpyDeviceToHost,
                       s));
    CK(cudaStreamSynchronize(s));
    const hl_result_hdr *hdr = reinterpret_cast<const hl_result_hdr *>(h->h_result);
    if (hdr->status != 0) {
        reset_counters(h, s);
        return HL_CUDA_ERROR;
    }
    int cnt = hdr->count;
    if (cnt > 0 && lines)
        memcpy(lines, h->h_result + sizeof(hl_result_hdr),
               sizeof(hl_line) * (size_t)cnt);
    *linesmax = cnt;
    return HL_NO_ERROR;
}

static int plain_launch(hl_handle *h, const hl_image_desc *img, int linesmax,
                        hl_line *lines_dev, int *count_dev, cudaStream_t s,
                        int ref_numrho_override = 0)
{
    hl_roi roi;
    int rc = roi_of(img, &roi);
    if (rc != HL_NO_ERROR)
        return rc;
    hl_geom g;
    if ((rc = hl_geometry(h, roi.w, roi.h, &g)) != HL_NO_ERROR)
        return rc;
    if (ref_numrho_override > 0)
        g.ref_numrho = ref_numrho_override;
    if ((rc = ensure_image(h, g, roi.w, roi.h, s)) != HL_NO_ERROR)
        return rc;
    if ((rc = ensure_acc(h, g.numrho, linesmax)) != HL_NO_ERROR)
        return rc;
    int launches = 0;
    h->last_batch = 0;
    if (!h->win_rows_override && !h->threads_override && !h->prof &&
        hl_small_fits(h->T, h->Tp, g.numrho)) {
        /* a small image: the whole path in one cluster launch, the
         * accumulator in shared memory only */
        hl_small_args sa;
        memset(&sa, 0, sizeof(sa));
        sa.roi = roi;
        sa.pts = reinterpret_cast<float2 *>(h->d_pts);
        sa.cosv = h->d_cos;
        sa.sinv = h->d_sin;
        sa.T = h->T;
        sa.Tp = h->Tp;
        sa.R = g.numrho;
        sa.rho_min = g.rho_min;
        sa.irho = (float)(1.0 / h->p.derho);   /* okano_3_0/HoughLine.cu:107 */
        sa.threshold = h->p.threshold;
        final_args(h, g, linesmax, lines_dev, count_dev, &sa.fin);
        sa.scale = (float)(1.0 / (h->T + 2));  /* :882-883 */
        CK(hl_launch_small(&sa, s));
        h->last_launches = 1;
        return HL_NO_ERROR;
    }
    if ((rc = run_ab(h, roi, g, true, s, &launches)) != HL_NO_ERROR)
        return rc;
    rc = run_c(h, g, !h->plan->add, linesmax, lines_dev, count_dev, s, &launches);
    h->last_launches = launches;
    return rc;
}

extern "C" int hl_plain(hl_handle *h, const hl_image_desc *img, int *linesmax,
                        hl_line *lines, void *stream)
{
    if (!h || !img || !linesmax)
        return HL_NULL_POINTER;
    if (*linesmax > 0 && !lines)
        return HL_NULL_POINTER;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    int rc = plain_launch(h, img, *linesmax, nullptr, nullptr, s);
    if (rc != HL_NO_ERROR)
        return rc;
    return fetch_result(h, linesmax, lines, s);
}

extern "C" int hl_plain_async(hl_handle *h, const hl_image_desc *img,
                              int linesmax, hl_line *lines_dev, int *count_dev,
                              void *stream)
{
    if (!h || !img)
        return HL_NULL_POINTER;
    if (linesmax > 0 && !lines_dev)
        return HL_NULL_POINTER;
    return plain_launch(h, img, linesmax, lines_dev, count_dev,
                        reinterpret_cast<cudaStream_t>(stream));
}

static int batch_last_status(hl_handle *h, int *status, cudaStream_t s);

extern "C" int hl_last_status(hl_handle *h, int *status, void *stream)
{
    if (!h || !status)
        return HL_NULL_POINTER;
    hl_result_hdr hdr;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (h->last_batch)
        return batch_last_status(h, status, s);
    if (!h->d_result) {
        *status = 0;
        return HL_NO_ERROR;
    }
    CK(cudaMemcpyAsync(&hdr, h->d_result, sizeof(hdr), cudaMemcpyDeviceToHost,
                       s));
    CK(cudaStreamSynchronize(s));
    *status = hdr.status;
    if (hdr.status != 0)
        reset_counters(h, s);
    return HL_NO_ERROR;
}

extern "C" int hl_compact(hl_handle *h, const hl_image_desc *img,
                          uint32_t *pts_dev, int *tile_off_dev, int *count_dev,
                          void *stream)
{
    if (!h || !img || !pts_dev || !tile_off_dev || !count_dev)
        return HL_NULL_POINTER;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    hl_roi roi;
    int rc = roi_of(img, &roi);
    if (rc != HL_NO_ERROR)
        return rc;
    hl_geom g;
    if ((rc = hl_geometry(h, roi.w, roi.h, &g)) != HL_NO_ERROR)
        return rc;
    if ((rc = ensure_image(h, g, roi.w, roi.h, s)) != HL_NO_ERROR)
        return rc;
    const int ntiles = g.tiles_x * g.tiles_y;
    hl_compact_args ca;
    memset(&ca, 0, sizeof(ca));
    ca.roi = roi;
    ca.tiles_x = g.tiles_x;
    ca.ntiles = ntiles;
    ca.imgs = nullptr;
    ca.group_img = nullptr;
    ca.nimg = 0;
    ca.ngroups = 0;
    ca.tile_state = h->d_tile_state;
    ca.ticket = reinterpret_cast<unsigned *>(h->d_counters + 3);
    ca.ticket_base = h->ticket_base;
    if (++h->epoch >= (1u << 30)) {
        CK(cudaMemsetAsync(h->d_tile_state, 0,
                           sizeof(unsigned long long) * h->cap_tiles, s));
        h->epoch = 1;
    }
    ca.epoch = h->epoch;
    ca.pts = pts_dev;
    ca.pts_f2 = nullptr;
    ca.tile_off = tile_off_dev;
    ca.count = count_dev;
    ca.status = h->d_counters + 1;
    {
        /* about one CTA per SM when they fit at once, else one per group */
        const int nct = hl_compact_persist_ctas(ntiles, h->sms);
        if (nct > 0) {
            CK(hl_launch_compact_persist(&ca, nct, s));
            h->ticket_base += (unsigned)nct;
        } else {
            CK(launch_compact_groups(h, &ca, s));
        }
    }
    h->last_launches = 1;
    return HL_NO_ERROR;
}

extern "C" int hl_accumulator(hl_handle *h, const hl_image_desc *img,
                              int32_t *acc_dev, void *stream)
{
    if (!h || !img || !acc_dev)
        return HL_NULL_POINTER;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    hl_roi roi;
    int rc = roi_of(img, &roi);
    if (rc != HL_NO_ERROR)
        return rc;
    hl_geom g;
    if ((rc = hl_geometry(h, roi.w, roi.h, &g)) != HL_NO_ERROR)
        return rc;
    if ((rc = ensure_image(h, g, roi.w, roi.h, s)) != HL_NO_ERROR)
        return rc;
    if ((rc = ensure_acc(h, g.numrho, 1)) != HL_NO_ERROR)
        return rc;
    int launches = 0;
    if ((rc = run_ab(h, roi, g, false, s, &launches)) != HL_NO_ERROR)
        return rc;
    CK(hl_launch_to_tight(h->d_acc, g.numrho, h->T, h->Tp, acc_dev, s));
    h->last_launches = launches + 1;
    return HL_NO_ERROR;
}

extern "C" int hl_accumulator_ref_layout(hl_handle *h, const hl_image_desc *img,
                                         int32_t *ref_dev, void *stream)
{
    if (!h || !img || !ref_dev)
        return HL_NULL_POINTER;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    hl_roi roi;
    int rc = roi_of(img, &roi);
    if (rc != HL_NO_ERROR)
        return rc;
    hl_geom g;
    if ((rc = hl_geometry(h, roi.w, roi.h, &g)) != HL_NO_ERROR)
        return rc;
    if ((rc = ensure_image(h, g, roi.w, roi.h, s)) != HL_NO_ERROR)
        return rc;
    if ((rc = ensure_acc(h, g.numrho, 1)) != HL_NO_ERROR)
        return rc;
    int launches = 0;
    if ((rc = run_ab(h, roi, g, false, s, &launches)) != HL_NO_ERROR)
        return rc;
    CK(hl_launch_to_ref(h->d_acc, g.numrho, h->T, h->Tp, g.rho_min,
                        g.ref_numrho, ref_dev, s));
    h->last_launches = launches + 1;
    return HL_NO_ERROR;
}

extern "C" int hl_lines_from_accumulator(hl_handle *h, const int32_t *acc_dev,
                                         int w, int hh, int *linesmax,
                                         hl_line *lines, void *stream)
{
    if (!h || !acc_dev || !linesmax)
        return HL_NULL_POINTER;
    if (*linesmax > 0 && !lines)
        return HL_NULL_POINTER;
    hl_geom g;
    int rc = hl_geometry(h, w, hh, &g);
    if (rc != HL_NO_ERROR)
        return rc;
    if ((rc = ensure_acc(h, g.numrho, *linesmax)) != HL_NO_ERROR)
        return rc;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    h->acc_state = ACC_ANY;
    CK(hl_launch_from_tight(acc_dev, g.numrho, h->T, h->Tp, h->d_acc, s));
    h->prof_open = 0;
    int launches = 1;
    if ((rc = run_c(h, g, false, *linesmax, nullptr, nullptr, s, &launches)) !=
        HL_NO_ERROR)
        return rc;
    h->last_launches = launches;
    return fetch_result(h, linesmax, lines, s);
}

/* Rows of the widest rho range a theta slice reaches over the box [x0, x1] x
 * [y0, y1] (in double, two rows of slack an end for the vote rule's floats and
 * 2^-20 of the value). */
static int points_span(const hl_handle *h, const int bb[4], int R)
{
    const double irho = (double)(float)(1.0 / h->p.derho);
    double span = 0.0;
    for (int k0 = 0; k0 < h->T; k0 += HL_SLICE) {
        double lo = 1e300, hi = -1e300;
        for (int k = k0; k < std::min(k0 + HL_SLICE, h->T); k++) {
            const double c = h->h_cos[k] * irho, s = h->h_sin[k] * irho;
            const double xa = bb[0] * c, xb = bb[2] * c, ya = bb[1] * s, yb = bb[3] * s;
            lo = std::min(lo, std::min(xa, xb) + std::min(ya, yb));
            hi = std::max(hi, std::max(xa, xb) + std::max(ya, yb));
        }
        const double slack = 3.0 + std::max(fabs(lo), fabs(hi)) / 1048576.0;
        span = std::max(span, hi - lo + 2.0 * slack);
    }
    return (int)std::min(span, (double)R);
}

extern "C" int hl_plain_points(hl_handle *h, const int *xy_dev, int n,
                               int *linesmax, hl_line *lines, void *stream)
{
    if (!h || !xy_dev || !linesmax)
        return HL_NULL_POINTER;
    if (*linesmax > 0 && !lines)
        return HL_NULL_POINTER;
    if (n <= 0)
        return HL_INVALID_DATA;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (!h->d_bbox)
        CK(cudaMalloc(&h->d_bbox, sizeof(int4) * HL_BBOX_CTAS));
    if (!h->h_bbox)
        CK(cudaMallocHost(&h->h_bbox, sizeof(int4)));
    CK(hl_launch_bbox(xy_dev, n, h->d_bbox, reinterpret_cast<unsigned *>(h->d_counters + 4),
                      h->h_bbox, s));
    CK(cudaStreamSynchronize(s));
    const int bb[4] = {h->h_bbox[0], h->h_bbox[1], h->h_bbox[2], h->h_bbox[3]};
    /* the reference's accumulator height uses the box extent,
     * okano_3_0/HoughLine.cu:374-375,387 */
    int w = bb[2] - bb[0], hh = bb[3] - bb[1];
    double ax = std::max(fabs((double)bb[0]), fabs((double)bb[2]));
    double ay = std::max(fabs((double)bb[1]), fabs((double)bb[3]));
    hl_geom g;
    g.numtheta = h->T;
    g.theta_pad = h->Tp;
    layout(h, sqrt(ax * ax + ay * ay) + 1.0, &g.rho_min, &g.numrho);
    g.ref_numrho = (int)((double)(int)((w + hh) * 2 + 1) / h->p.derho);
    if ((double)g.numrho * h->Tp >= 2147483647.0)
        return HL_OP_OVERFLOW;
    int rc = ensure_acc(h, g.numrho, *linesmax);
    if (rc != HL_NO_ERROR)
        return rc;
    hl_points_args pa;
    memset(&pa, 0, sizeof(pa));
    pa.xy = reinterpret_cast<const int2 *>(xy_dev);
    pa.n = n;
    pa.x0 = bb[0];
    pa.y0 = bb[1];
    pa.x1 = bb[2];
    pa.y1 = bb[3];
    pa.cosv = h->d_cos;
    pa.sinv = h->d_sin;
    pa.T = h->T;
    pa.Tp = h->Tp;
    pa.rho_min = g.rho_min;
    pa.R = g.numrho;
    pa.span = points_span(h, bb, g.numrho);
    pa.exact = g.numrho >= (1 << 22);
    pa.irho = (float)(1.0 / h->p.derho);
    pa.acc = h->d_acc;
    h->acc_state = ACC_ANY;
    CK(hl_launch_vote_points(&pa, std::max(h->sms, 1), s));
    int launches = 2;
    h->prof_open = 0;
    if ((rc = run_c(h, g, false, *linesmax, nullptr, nullptr, s, &launches)) !=
        HL_NO_ERROR)
        return rc;
    h->last_launches = launches;
    return fetch_result(h, linesmax, lines, s);
}

extern "C" int hl_measure_smem_atomic_peak(int iters, double *atomics_per_s,
                                           void *stream)
{
    if (!atomics_per_s)
        return HL_NULL_POINTER;
    if (iters <= 0)
        return HL_INVALID_DATA;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    int *sink = nullptr;
    CK(cudaMalloc(&sink, sizeof(int)));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int blocks = 0, threads = 0;
    cudaError_t e = hl_launch_atomic_bench(iters / 4 + 1, sink, s, &blocks,
                                           &threads);   /* warm-up */
    float best = 1e30f;
    for (int rep = 0; rep < 3 && e == cudaSuccess; rep++) {
        cudaEventRecord(e0, s);
        e = hl_launch_atomic_bench(iters, sink, s, &blocks, &threads);
        cudaEventRecord(e1, s);
        if (e == cudaSuccess)
            e = cudaEventSynchronize(e1);
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        best = std::min(best, ms);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(sink);
    if (e != cudaSuccess)
        return map_err(e);
    double total = (double)blocks * threads * (double)iters * 8.0;
    *atomics_per_s = total / (best * 1e-3);
    return HL_NO_ERROR;
}

extern "C" int hl_plain_draw(hl_handle *h, const hl_image_desc *in,
                             const hl_image_desc *out, int *linesmax,
                             hl_line *lines, void *stream)
{
    if (!h || !in || !out || !linesmax || !out->data)
        return HL_NULL_POINTER;
    if (*linesmax > 0 && !lines)
        return HL_NULL_POINTER;
    hl_roi rin, rout;
    int rc = roi_of(in, &rin);
    if (rc != HL_NO_ERROR)
        return rc;
    if ((rc = roi_of(out, &rout)) != HL_NO_ERROR)
        return rc;
    /* okano_3_0/HoughLine.cu:1101-1109: both ROIs shrink to the smaller
     * width and height; the accumulator height still comes from the input
     * ROI (:670), which only the decode sees */
    const int ref_nrho = (int)((double)(int)((rin.w + rin.h) * 2 + 1) / h->p.derho);
    const int w = std::min(rin.w, rout.w), hh = std::min(rin.h, rout.h);
    hl_image_desc vin = *in;
    vin.roi_x2 = vin.roi_x1 + w;
    vin.roi_y2 = vin.roi_y1 + hh;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    rc = plain_launch(h, &vin, *linesmax, nullptr, nullptr, s, ref_nrho);
    if (rc != HL_NO_ERROR)
        return rc;
    const int launches = h->last_launches;
    /* the drawing kernel reads the records in the device result block; with
     * room for few lines it is queued behind the tail and takes the count
     * from the block, so the call waits once */
    const hl_line *dl = reinterpret_cast<const hl_line *>(h->d_result + sizeof(hl_result_hdr));
    const int derho_i = (int)h->p.derho;   /* _houghoutKer takes an int derho */
    const bool queued = derho_i != 0 && *linesmax > 0 && *linesmax <= 1024;
    if (queued)
        CK(hl_launch_draw(const_cast<uint8_t *>(rout.base), rout.pitch, w, hh, dl, *linesmax,
                          reinterpret_cast<const hl_result_hdr *>(h->d_result), derho_i, s));
    rc = fetch_result(h, linesmax, lines, s);
    if (rc != HL_NO_ERROR)
        return rc;
    if (*linesmax > 0) {
        if (derho_i == 0)
            return HL_INVALID_DATA;
        if (!queued) {
            CK(hl_launch_draw(const_cast<uint8_t *>(rout.base), rout.pitch, w, hh, dl,
                              *linesmax, nullptr, derho_i, s));
            CK(cudaStreamSynchronize(s));
        }
        h->last_launches = launches + (*linesmax + HL_DRAW_LINES - 1) / HL_DRAW_LINES;
    }
    return HL_NO_ERROR;
}

extern "C" int hl_draw_lines(hl_handle *h, const hl_image_desc *out,
                             const hl_line *lines, int nlines, void *stream)
{
    if (!h || !out)
        return HL_NULL_POINTER;
    if (nlines <= 0)
        return HL_NO_ERROR;
    if (!lines)
        return HL_NULL_POINTER;
    hl_roi r;
    int rc = roi_of(out, &r);
    if (rc != HL_NO_ERROR)
        return rc;
    int derho_i = (int)h->p.derho;
    if (derho_i == 0)
        return HL_INVALID_DATA;
    size_t bytes = sizeof(hl_result_hdr) + sizeof(hl_line) * (size_t)nlines;
    if ((rc = grow((void **)&h->d_aux, &h->cap_aux, bytes)) != HL_NO_ERROR)
        return rc;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    CK(cudaMemcpyAsync(h->d_aux, lines, sizeof(hl_line) * (size_t)nlines,
                       cudaMemcpyHostToDevice, s));
    CK(hl_launch_draw(const_cast<uint8_t *>(r.base), r.pitch, r.w, r.h,
                      reinterpret_cast<const hl_line *>(h->d_aux), nlines, nullptr,
                      derho_i, s));
    CK(cudaStreamSynchronize(s));
    h->last_launches = (nlines + HL_DRAW_LINES - 1) / HL_DRAW_LINES;
    return HL_NO_ERROR;
}

extern "C" int hl_real_line(hl_handle *h, const hl_image_desc *img, int x1,
                            int y1, int x2, int y2, float threshold,
                            float thresperc, int *is_real, int *pointnum,
                            void *stream)
{
    if (!h || !img || !is_real)
        return HL_NULL_POINTER;
    hl_roi roi;
    int rc = roi_of(img, &roi);
    if (rc != HL_NO_ERROR)
        return rc;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    int *cnt = h->d_counters + 8;
    CK(cudaMemsetAsync(cnt, 0, sizeof(int), s));
    /* okano_3_0/HoughLine.cu:1436-1443: the float threshold is passed to an
     * int parameter (truncation) */
    CK(hl_launch_real_line(roi.base, roi.pitch, roi.w, roi.h, x1, y1, x2, y2,
                           (int)threshold, cnt, s));
    int n = 0;
    CK(cudaMemcpyAsync(&n, cnt, sizeof(int), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    /* :1405: int pointnumfull = sqrt(0.0 + dx*dx + dy*dy) */
    const int full = (int)sqrt(0.0 + (double)(x1 - x2) * (x1 - x2) +
                               (double)(y1 - y2) * (y1 - y2));
    *is_real = ((float)n > (float)full * thresperc) ? 1 : 0;
    if (pointnum)
        *pointnum = n;
    h->last_launches = 1;
    return HL_NO_ERROR;
}

/* ==================================================================== */
/* Batched path                                                          */
/* ==================================================================== */

/* Counters of a batch call, cleared at its start: [0] compaction ticket,
 * [1] vote work counter, [2] status word, [3] total points, [8] noted peak
 * candidates. */
#define BW_NCNT 16

struct hl_batch_ws {
    float2 *d_pts;
    size_t cap_pts;
    unsigned long long *d_state;   /* look-back state per 4-tile group */
    size_t cap_state;
    int *d_tile_off;
    size_t cap_tile_off;
    int32_t *d_acc;
    size_t cap_acc;
    unsigned long long *d_keys;
    size_t cap_keys;
    unsigned long long *d_cand;    /* noted peak candidates; counter d_cnt[8] */
    size_t cap_cand;
    unsigned char *d_scratch;      /* the vote items' slabs */
    size_t cap_scratch;
    int *d_ncand;                  /* per image, zero between calls */
    size_t cap_ncand;
    int *d_cnt;
    unsigned char *d_tab;          /* per-image tables of one call */
    size_t cap_tab;
    unsigned char *h_tab;          /* their pinned staging copy */
    size_t cap_htab;
    hl_line *d_lines;              /* hl_batch's device results */
    size_t cap_lines;
    int *d_counts;
    size_t cap_counts;
    unsigned char *h_res;          /* pinned copy of results + status */
    size_t cap_hres;
    cudaEvent_t tab_read;          /* the previous call's table upload */
    int tab_event;

    /* the plan of the last call (reused while the geometry is the same) */
    std::vector<int> key;
    size_t tab_bytes;
    size_t off_cimg, off_gimg, off_vimg, off_plan, off_pimg, off_chunks, off_fimg;
    int ngroups, ntiles, nchunks, grid, threads;
    size_t npts_cap, acc_ints, nkeys;
    std::vector<size_t> acc_off, key_off;
    std::vector<size_t> pts_base;  /* each image's first point */
    std::vector<int> key_cap_i, tile_base, group_base, rho_min, R, ref_numrho;
    vote_plan plan;
    bool acc_zero;                 /* d_acc is zero between calls */
    std::vector<int2> chunks;
    std::vector<int> group_img;

    /* captured pipeline (captured on a private stream: the caller's may be
     * the legacy default stream, which cannot be captured) */
    cudaStream_t cap_stream;
    cudaGraphExec_t gexec;
    std::vector<long long> gkey;
};

static void batch_ws_free(hl_batch_ws *b);
static void prop_free(hl_handle *h);

static void batch_free(hl_handle *h)
{
    batch_ws_free(h->bw);
    batch_ws_free(h->bw_fb);
    h->bw = h->bw_fb = nullptr;
    prop_free(h);
}

static void batch_ws_free(hl_batch_ws *b)
{
    if (!b)
        return;
    void *dp[] = {b->d_pts, b->d_state, b->d_tile_off, b->d_acc, b->d_keys, b->d_cand,
                  b->d_ncand, b->d_cnt, b->d_tab, b->d_lines, b->d_counts,
                  b->d_scratch};
    for (void *q : dp)
        if (q)
            cudaFree(q);
    if (b->h_tab)
        cudaFreeHost(b->h_tab);
    if (b->h_res)
        cudaFreeHost(b->h_res);
    if (b->tab_event)
        cudaEventDestroy(b->tab_read);
    if (b->gexec)
        cudaGraphExecDestroy(b->gexec);
    if (b->cap_stream)
        cudaStreamDestroy(b->cap_stream);
    delete b;
}

static size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }

/* the launch's grid and the places of its tables */
static void batch_layout(const hl_handle *h, hl_batch_ws *b, int nimg)
{
    b->grid = std::max(1, std::min((int)b->plan.items.size(),
                                   vote_ctas(h, b->plan.win_rows, b->threads)));
    size_t o = 0;
    b->off_cimg = o;   o = align16(o + sizeof(hl_compact_img) * nimg);
    b->off_gimg = o;   o = align16(o + sizeof(int) * (size_t)b->ngroups);
    b->off_vimg = o;   o = align16(o + sizeof(hl_vote_img) * nimg);
    b->off_plan = o;   o = align16(o + plan_bytes(b->plan));
    b->off_pimg = o;   o = align16(o + sizeof(hl_peak_img) * nimg);
    b->off_chunks = o; o = align16(o + sizeof(int2) * b->chunks.size());
    b->off_fimg = o;   o = align16(o + sizeof(hl_final_img) * nimg);
    b->tab_bytes = o;
}

/* Plan a batch: sizes, offsets, work items, chunks; fills the pinned tables
 * (image pointers and thresholds included).  The geometry part is reused
 * when the sizes and the launch shape equal the previous call's.  src: the
 * points are another workspace's, image i's those of its image src_img[i]. */
static int batch_plan(hl_handle *h, hl_batch_ws *b, const hl_image_desc *imgs,
                      int nimg, const int *thr, int K, hl_line *lines_dev,
                      int *counts_dev, const hl_roi *rois, cudaStream_t s,
                      const hl_batch_ws *src = nullptr, const int *src_img = nullptr)
{
    std::vector<hl_geom> gs((size_t)nimg);
    for (int i = 0; i < nimg; i++) {
        int rc = hl_geometry(h, rois[i].w, rois[i].h, &gs[i]);
        if (rc != HL_NO_ERROR)
            return rc;
    }
    /* launch shape: the override (autotuner) or the largest window that
     * fits, 1024 threads */
    const int cap = plan_cap(h), threads = vote_threads(h);

    std::vector<int> key;
    key.reserve(2 * (size_t)nimg + 8);
    key.push_back(nimg);
    key.push_back(cap);
    key.push_back(threads);
    key.push_back(h->T);
    for (double v : {h->p.derho, h->p.detheta}) {   /* rho range, theta table */
        unsigned long long bits;
        memcpy(&bits, &v, sizeof(bits));
        key.push_back((int)(bits & 0xffffffffu));
        key.push_back((int)(bits >> 32));
    }
    for (int i = 0; i < nimg; i++) {
        key.push_back(rois[i].w);
        key.push_back(rois[i].h);
    }
    if (key != b->key) {
        b->key.clear();   /* not valid until the plan below is whole */
        b->threads = threads;
        b->acc_off.assign(nimg, 0);
        b->key_off.assign(nimg, 0);
        b->key_cap_i.assign(nimg, 0);
        b->tile_base.assign(nimg, 0);
        b->group_base.assign(nimg, 0);
        b->rho_min.assign(nimg, 0);
        b->R.assign(nimg, 0);
        b->ref_numrho.assign(nimg, 0);
        b->group_img.clear();
        b->chunks.clear();
        size_t acc = 0, keys = 0, pts = 0;
        b->pts_base.assign(nimg, 0);
        int tiles = 0, groups = 0;
        std::vector<plan_img> pim((size_t)nimg);
        for (int i = 0; i < nimg; i++) {
            const hl_geom &g = gs[i];
            const int nt = g.tiles_x * g.tiles_y;
            const int ng = (nt + HL_COMPACT_GROUP - 1) / HL_COMPACT_GROUP;
            b->tile_base[i] = tiles;
            b->group_base[i] = groups;
            for (int q = 0; q < ng; q++)
                b->group_img.push_back(i);
            tiles += nt + 1;   /* the image's tile offsets and its end */
            groups += ng;
            /* room for every pixel and one pad per tile, kept even so every
             * image's point list starts on 16 bytes */
            b->pts_base[i] = pts;
            pts += ((size_t)rois[i].w * rois[i].h + (size_t)nt + 16 + 1) & ~(size_t)1;
            b->acc_off[i] = acc;
            acc += (size_t)g.numrho * h->Tp;
            /* peak-key capacity: the bound of ensure_acc, at most 2^17 */
            const size_t kc = std::min((size_t)g.numrho * ((h->T + 1) / 2) + 32,
                                       (size_t)1 << 17);
            b->key_off[i] = keys;
            b->key_cap_i[i] = (int)kc;
            keys += kc;
            b->rho_min[i] = g.rho_min;
            b->R[i] = g.numrho;
            b->ref_numrho[i] = g.ref_numrho;
            pim[i] = {rois[i].w, rois[i].h, g.numrho, g.rho_min};
            for (int r0 = 0; r0 < g.numrho; r0 += HL_PEAK_ROWS)
                b->chunks.push_back(make_int2(i, r0));
        }
        if (nimg > 0xffff)
            return HL_OP_OVERFLOW;
        int rc = make_plan(h, pim.data(), nimg, cap, std::max(h->sms, 1), true, &b->plan);
        if (rc != HL_NO_ERROR)
            return rc;
        b->ngroups = groups;
        b->ntiles = tiles;
        b->nchunks = (int)b->chunks.size();
        b->npts_cap = pts;
        b->acc_ints = acc;
        b->nkeys = keys;
        batch_layout(h, b, nimg);
        b->key = key;
    }

    /* device buffers */
    int rc;
    if (b->cap_acc < sizeof(int32_t) * b->acc_ints)
        b->acc_zero = false;   /* another buffer, also after a failed allocation */
    if ((!src &&
         ((rc = grow((void **)&b->d_pts, &b->cap_pts, sizeof(float2) * b->npts_cap)) !=
              HL_NO_ERROR ||
          (rc = grow((void **)&b->d_state, &b->cap_state,
                     sizeof(unsigned long long) * ((size_t)b->ngroups + 1))) != HL_NO_ERROR ||
          (rc = grow((void **)&b->d_tile_off, &b->cap_tile_off,
                     sizeof(int) * ((size_t)b->ntiles + 1))) != HL_NO_ERROR)) ||
        (rc = grow((void **)&b->d_acc, &b->cap_acc, sizeof(int32_t) * b->acc_ints)) != HL_NO_ERROR ||
        (rc = grow((void **)&b->d_cand, &b->cap_cand,
                   sizeof(unsigned long long) * (65536 + b->acc_ints / 128))) != HL_NO_ERROR ||
        (rc = grow((void **)&b->d_keys, &b->cap_keys,
                   sizeof(unsigned long long) * b->nkeys)) != HL_NO_ERROR ||
        (rc = grow((void **)&b->d_tab, &b->cap_tab, b->tab_bytes)) != HL_NO_ERROR)
        return rc;
    rc = grow((void **)&b->d_scratch, &b->cap_scratch, plan_scratch(b->plan));
    if (rc == HL_OUT_OF_MEM && !b->plan.add) {
        /* no room for the slabs: the form without them, whose tables are smaller */
        std::vector<plan_img> pim((size_t)nimg);
        for (int i = 0; i < nimg; i++)
            pim[i] = {rois[i].w, rois[i].h, b->R[i], b->rho_min[i]};
        b->key.clear();
        if ((rc = make_plan(h, pim.data(), nimg, cap, std::max(h->sms, 1), false, &b->plan)) !=
            HL_NO_ERROR)
            return rc;
        batch_layout(h, b, nimg);
        b->key = key;
        rc = grow((void **)&b->d_scratch, &b->cap_scratch, plan_scratch(b->plan));
    }
    if (rc != HL_NO_ERROR)
        return rc;
    if (b->cap_ncand < sizeof(int) * (size_t)nimg || !b->d_ncand) {
        if ((rc = grow((void **)&b->d_ncand, &b->cap_ncand, sizeof(int) * (size_t)nimg)) !=
            HL_NO_ERROR)
            return rc;
        CK(cudaMemsetAsync(b->d_ncand, 0, b->cap_ncand, s));   /* not the default stream's */
    }
    if (!b->d_cnt)
        CK(cudaMalloc(&b->d_cnt, BW_NCNT * sizeof(int)));
    /* the previous call's upload must be done before the staging is reused */
    if (b->tab_event)
        CK(cudaEventSynchronize(b->tab_read));
    if ((rc = grow_host(&b->h_tab, &b->cap_htab, b->tab_bytes)) != HL_NO_ERROR)
        return rc;

    /* tables */
    unsigned char *t = b->h_tab;
    hl_compact_img *ci = reinterpret_cast<hl_compact_img *>(t + b->off_cimg);
    hl_vote_img *vi = reinterpret_cast<hl_vote_img *>(t + b->off_vimg);
    hl_peak_img *pi = reinterpret_cast<hl_peak_img *>(t + b->off_pimg);
    hl_final_img *fi = reinterpret_cast<hl_final_img *>(t + b->off_fimg);
    for (int i = 0; i < nimg; i++) {
        const hl_geom &g = gs[i];
        const int nt = g.tiles_x * g.tiles_y;
        ci[i].roi = rois[i];
        ci[i].tiles_x = g.tiles_x;
        ci[i].ntiles = nt;
        ci[i].tile_base = b->tile_base[i];
        ci[i].group_base = b->group_base[i];
        ci[i].ngroups = (nt + HL_COMPACT_GROUP - 1) / HL_COMPACT_GROUP;
        ci[i].pad = 0;
        ci[i].pts_base = (long long)b->pts_base[i];
        vi[i].pts = src ? src->d_pts + src->pts_base[(size_t)src_img[i]]
                        : b->d_pts + b->pts_base[i];
        vi[i].tile_off = src ? src->d_tile_off + src->tile_base[(size_t)src_img[i]]
                             : b->d_tile_off + b->tile_base[i];
        vi[i].ntiles = nt;
        vi[i].tiles_x = g.tiles_x;
        vi[i].w = rois[i].w;
        vi[i].h = rois[i].h;
        vi[i].rho_min = g.rho_min;
        vi[i].R = g.numrho;
        vi[i].threshold = thr ? thr[i] : h->p.threshold;
        vi[i].pad = 0;
        vi[i].acc = b->d_acc + b->acc_off[i];
        pi[i].acc = b->d_acc + b->acc_off[i];
        pi[i].keys = b->d_keys + b->key_off[i];
        pi[i].ncand = b->d_ncand + i;
        pi[i].R = g.numrho;
        pi[i].cap = b->key_cap_i[i];
        pi[i].threshold = thr ? thr[i] : h->p.threshold;
        pi[i].pad = 0;
        fi[i].keys = b->d_keys + b->key_off[i];
        fi[i].ncand = b->d_ncand + i;
        fi[i].cap = b->key_cap_i[i];
        fi[i].rho_min = g.rho_min;
        fi[i].ref_numrho = g.ref_numrho;
        fi[i].pad = 0;
        fi[i].lines = lines_dev + (size_t)i * (size_t)std::max(K, 0);
        fi[i].count_out = counts_dev + i;
    }
    memcpy(t + b->off_gimg, b->group_img.data(), sizeof(int) * b->group_img.size());
    plan_copy(b->plan, t + b->off_plan);
    memcpy(t + b->off_chunks, b->chunks.data(), sizeof(int2) * b->chunks.size());
    return HL_NO_ERROR;
}

/* The stream work of one planned batch call. */
/* counters, look-back states, tables, then the compaction of every image */
static int batch_enqueue_compact(hl_handle *h, hl_batch_ws *b, int nimg,
                                 cudaStream_t s)
{
    unsigned char *dt = b->d_tab;
    CK(cudaMemsetAsync(b->d_cnt, 0, BW_NCNT * sizeof(int), s));
    CK(cudaMemsetAsync(b->d_state, 0,
                       sizeof(unsigned long long) * ((size_t)b->ngroups + 1), s));
    CK(cudaMemcpyAsync(dt, b->h_tab, b->tab_bytes, cudaMemcpyHostToDevice, s));

    hl_compact_args ca;
    memset(&ca, 0, sizeof(ca));
    ca.imgs = reinterpret_cast<const hl_compact_img *>(dt + b->off_cimg);
    ca.group_img = reinterpret_cast<const int *>(dt + b->off_gimg);
    ca.nimg = nimg;
    ca.ngroups = b->ngroups;
    ca.tile_state = b->d_state;
    ca.ticket = reinterpret_cast<unsigned *>(b->d_cnt + 0);
    ca.ticket_base = 0;
    ca.epoch = 1;
    ca.pts = nullptr;
    ca.pts_f2 = b->d_pts;
    ca.tile_off = b->d_tile_off;
    ca.count = b->d_cnt + 3;
    ca.status = b->d_cnt + 2;
    CK(hl_launch_compact(&ca, s));
    prof_mark(h, 1, s);
    return HL_NO_ERROR;
}

/* the full vote and the peak pass */
static int batch_enqueue_vote_peaks(hl_handle *h, hl_batch_ws *b, cudaStream_t s)
{
    unsigned char *dt = b->d_tab;
    hl_vote_args va;
    memset(&va, 0, sizeof(va));
    va.imgs = reinterpret_cast<const hl_vote_img *>(dt + b->off_vimg);
    va.cosv = h->d_cos;
    va.sinv = h->d_sin;
    va.T = h->T;
    va.Tp = h->Tp;
    va.irho = (float)(1.0 / h->p.derho);   /* okano_3_0/HoughLine.cu:107 */
    va.status = b->d_cnt + 2;
    /* the counter is cleared with the others at the start of every call */
    va.cand = b->plan.add ? cand_list(nullptr, 0, nullptr)
                          : cand_list(b->d_cand, b->cap_cand, b->d_cnt + 8);
    va.work = reinterpret_cast<unsigned *>(b->d_cnt + 1);
    va.work_base = 0;
    hl_merge_args ma;
    memset(&ma, 0, sizeof(ma));
    plan_args(b->plan, dt + b->off_plan, b->d_scratch, &va, &ma);
    if (va.add)
        CK(cudaMemsetAsync(b->d_acc, 0, sizeof(int32_t) * b->acc_ints, s));
    CK(hl_launch_vote(&va, b->threads, b->grid, s));
    if (ma.nblocks > 0)
        CK(hl_launch_merge(&ma, s));
    prof_mark(h, 2, s);

    hl_peak_args pa;
    memset(&pa, 0, sizeof(pa));
    pa.imgs = reinterpret_cast<const hl_peak_img *>(dt + b->off_pimg);
    pa.chunks = reinterpret_cast<const int2 *>(dt + b->off_chunks);
    pa.nchunks = b->nchunks;
    pa.T = h->T;
    pa.Tp = h->Tp;
    pa.status = b->d_cnt + 2;
    pa.cand = va.cand;
    CK(hl_launch_peaks(&pa, s));
    prof_mark(h, 3, s);
    return HL_NO_ERROR;
}

/* rank, merge and write the lines of every image; voted: clear the bins that
 * the vote stored */
static int batch_enqueue_finalize(hl_handle *h, hl_batch_ws *b, int nimg, int K, bool voted,
                                  cudaStream_t s)
{
    unsigned char *dt = b->d_tab;
    hl_final_args fa;
    memset(&fa, 0, sizeof(fa));
    fa.imgs = reinterpret_cast<const hl_final_img *>(dt + b->off_fimg);
    fa.T = h->T;
    fa.detheta = h->p.detheta;
    fa.thresdis = h->p.thresdis;
    fa.thresang = h->p.thresang;
    fa.linesmax = K;
    fa.hdr = nullptr;
    fa.status = b->d_cnt + 2;
    if (voted && !b->plan.add) {
        fa.clear = cand_list(b->d_cand, b->cap_cand, b->d_cnt + 8);
        fa.clear_imgs = reinterpret_cast<const hl_peak_img *>(dt + b->off_pimg);
        fa.acc = b->d_acc;
        fa.acc_ints = (long long)b->acc_ints;
        fa.Tp = h->Tp;
    }
    CK(hl_launch_finalize(&fa, nimg, s));
    prof_mark(h, 4, s);
    return HL_NO_ERROR;
}

static int batch_enqueue(hl_handle *h, hl_batch_ws *b, int nimg, int K,
                         cudaStream_t s, const hl_batch_ws *src = nullptr)
{
    int rc;
    if (src) {
        /* counters and tables; the compaction's status with its points */
        CK(cudaMemsetAsync(b->d_cnt, 0, BW_NCNT * sizeof(int), s));
        CK(cudaMemcpyAsync(b->d_cnt + 2, src->d_cnt + 2, sizeof(int), cudaMemcpyDeviceToDevice,
                           s));
        CK(cudaMemcpyAsync(b->d_tab, b->h_tab, b->tab_bytes, cudaMemcpyHostToDevice, s));
        prof_mark(h, 1, s);
    } else if ((rc = batch_enqueue_compact(h, b, nimg, s)) != HL_NO_ERROR) {
        return rc;
    }
    if ((rc = batch_enqueue_vote_peaks(h, b, s)) != HL_NO_ERROR)
        return rc;
    return batch_enqueue_finalize(h, b, nimg, K, true, s);
}

/* src, src_img: see batch_plan (never captured: the points' places change) */
static int batch_run_ws(hl_handle *h, hl_batch_ws **pb, const hl_image_desc *imgs,
                        int nimg, const int *thr, int K, hl_line *lines_dev,
                        int *counts_dev, cudaStream_t s, const hl_batch_ws *src = nullptr,
                        const int *src_img = nullptr)
{
    if (nimg <= 0)
        return HL_INVALID_DATA;
    if (!*pb) {
        *pb = new (std::nothrow) hl_batch_ws();
        if (!*pb)
            return HL_OUT_OF_MEM;
    }
    hl_batch_ws *b = *pb;
    std::vector<hl_roi> rois((size_t)nimg);
    for (int i = 0; i < nimg; i++) {
        int rc = roi_of(&imgs[i], &rois[i]);
        if (rc != HL_NO_ERROR)
            return rc;
    }
    int rc = batch_plan(h, b, imgs, nimg, thr, K, lines_dev, counts_dev, rois.data(), s,
                        src, src_img);
    if (rc != HL_NO_ERROR)
        return rc;
    h->last_batch = 1;
    h->last_launches = src ? 3 : 4;
    if (!b->tab_event) {
        CK(cudaEventCreateWithFlags(&b->tab_read, cudaEventDisableTiming));
        b->tab_event = 1;
    }
    if (!b->acc_zero && !b->plan.add)   /* outside the (captured) pipeline */
        CK(cudaMemsetAsync(b->d_acc, 0, b->cap_acc, s));
    b->acc_zero = false;
    prof_mark(h, 0, s);
    if (!h->batch_graph || h->prof || src) {
        rc = batch_enqueue(h, b, nimg, K, s, src);
    } else {
        /* graph key: the plan key plus what the captured nodes hold */
        std::vector<long long> gk(b->key.begin(), b->key.end());
        const void *held[] = {lines_dev, counts_dev, h->d_cos, h->d_sin, b->d_acc, b->d_pts,
                              b->d_state, b->d_tile_off, b->d_tab, b->h_tab, b->d_keys,
                              b->d_ncand, b->d_cnt, b->d_scratch, b->d_cand};
        for (const void *p : held)
            gk.push_back((long long)(uintptr_t)p);
        unsigned ang;
        memcpy(&ang, &h->p.thresang, sizeof(ang));
        gk.push_back(K);
        gk.push_back(h->p.thresdis);
        gk.push_back((long long)ang);
        gk.push_back(b->plan.add);
        gk.push_back((long long)b->plan.items.size());
        if (!b->gexec || gk != b->gkey) {
            if (b->gexec) {
                cudaGraphExecDestroy(b->gexec);
                b->gexec = nullptr;
            }
            if (!b->cap_stream)
                CK(cudaStreamCreateWithFlags(&b->cap_stream, cudaStreamNonBlocking));
            cudaGraph_t graph = nullptr;
            CK(cudaStreamBeginCapture(b->cap_stream, cudaStreamCaptureModeThreadLocal));
            rc = batch_enqueue(h, b, nimg, K, b->cap_stream);
            cudaError_t e = cudaStreamEndCapture(b->cap_stream, &graph);
            if (rc != HL_NO_ERROR) {
                if (graph)
                    cudaGraphDestroy(graph);
                return rc;
            }
            if (e != cudaSuccess)
                return map_err(e);
            e = cudaGraphInstantiate(&b->gexec, graph, 0);
            cudaGraphDestroy(graph);
            if (e != cudaSuccess) {
                b->gexec = nullptr;
                return map_err(e);
            }
            b->gkey = gk;
        }
        CK(cudaGraphLaunch(b->gexec, s));
        h->last_launches = 4;
    }
    if (rc == HL_NO_ERROR) {
        b->acc_zero = !b->plan.add;   /* the tail clears what is stored */
        CK(cudaEventRecord(b->tab_read, s));
    }
    return rc;
}

static int batch_run(hl_handle *h, const hl_image_desc *imgs, int nimg,
                     const int *thr, int K, hl_line *lines_dev,
                     int *counts_dev, cudaStream_t s)
{
    return batch_run_ws(h, &h->bw, imgs, nimg, thr, K, lines_dev, counts_dev, s);
}

/* Every reader of a batch's status word comes here: after an error (a launch that
 * gave up) the accumulators are cleared before the next call relies on them. */
static int batch_status(hl_batch_ws *b, int status)
{
    if (status != 0)
        b->acc_zero = false;
    return status;
}

static int batch_last_status(hl_handle *h, int *status, cudaStream_t s)
{
    hl_batch_ws *b = h->bw;
    if (!b || !b->d_cnt) {
        *status = 0;
        return HL_NO_ERROR;
    }
    int st = 0;
    CK(cudaMemcpyAsync(&st, b->d_cnt + 2, sizeof(int), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    *status = batch_status(b, st);
    return HL_NO_ERROR;
}

extern "C" int hl_set_batch_graph(hl_handle *h, int enable)
{
    if (!h)
        return HL_NULL_POINTER;
    h->batch_graph = enable ? 1 : 0;
    return HL_NO_ERROR;
}

extern "C" int hl_batch_async(hl_handle *h, const hl_image_desc *imgs, int nimg,
                              const int *thresholds, int linesmax,
                              hl_line *lines_dev, int *counts_dev, void *stream)
{
    if (!h || !imgs || !counts_dev)
        return HL_NULL_POINTER;
    if (linesmax > 0 && !lines_dev)
        return HL_NULL_POINTER;
    return batch_run(h, imgs, nimg, thresholds, linesmax, lines_dev, counts_dev,
                     reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int hl_tiles(hl_handle *h, const hl_image_desc *img, int piecenum, int linesmax,
                        hl_line *lines, int *counts, void *stream)
{
    if (!h || !img || !counts)
        return HL_NULL_POINTER;
    if (piecenum <= 0 || piecenum > 1024)
        return HL_INVALID_DATA;
    const int cx = img->width / piecenum, cy = img->height / piecenum;
    if (cx < 2 || cy < 2)
        return HL_INVALID_DATA;
    std::vector<hl_image_desc> cells((size_t)piecenum * piecenum, *img);
    for (int y = 0; y < piecenum; y++)
        for (int x = 0; x < piecenum; x++) {
            hl_image_desc &d = cells[(size_t)y * piecenum + x];
            d.roi_x1 = x * cx;
            d.roi_x2 = x * cx + cx - 1;   /* okano_3_0/HoughRec.cu:745-748 */
            d.roi_y1 = y * cy;
            d.roi_y2 = y * cy + cy - 1;
        }
    return hl_batch(h, cells.data(), (int)cells.size(), nullptr, linesmax, lines, counts,
                    stream);
}

extern "C" int hl_batch(hl_handle *h, const hl_image_desc *imgs, int nimg,
                        const int *thresholds, int linesmax, hl_line *lines,
                        int *counts, void *stream)
{
    if (!h || !imgs || !counts)
        return HL_NULL_POINTER;
    if (linesmax > 0 && !lines)
        return HL_NULL_POINTER;
    if (nimg <= 0)
        return HL_INVALID_DATA;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (!h->bw) {
        h->bw = new (std::nothrow) hl_batch_ws();
        if (!h->bw)
            return HL_OUT_OF_MEM;
    }
    hl_batch_ws *b = h->bw;
    const size_t K = (size_t)std::max(linesmax, 0);
    int rc;
    if ((rc = grow((void **)&b->d_lines, &b->cap_lines,
                   sizeof(hl_line) * std::max(K * nimg, (size_t)1))) != HL_NO_ERROR ||
        (rc = grow((void **)&b->d_counts, &b->cap_counts, sizeof(int) * nimg)) != HL_NO_ERROR)
        return rc;
    rc = batch_run(h, imgs, nimg, thresholds, linesmax, b->d_lines, b->d_counts, s);
    if (rc != HL_NO_ERROR)
        return rc;
    const size_t lbytes = sizeof(hl_line) * K * nimg;
    if ((rc = grow_host(&b->h_res, &b->cap_hres, lbytes + sizeof(int) * (nimg + 1))) !=
        HL_NO_ERROR)
        return rc;
    int *h_counts = reinterpret_cast<int *>(b->h_res + lbytes);
    CK(cudaMemcpyAsync(h_counts, b->d_counts, sizeof(int) * nimg,
                       cudaMemcpyDeviceToHost, s));
    CK(cudaMemcpyAsync(h_counts + nimg, b->d_cnt + 2, sizeof(int),
                       cudaMemcpyDeviceToHost, s));
    if (lbytes)
        CK(cudaMemcpyAsync(b->h_res, b->d_lines, lbytes, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (batch_status(b, h_counts[nimg]) != 0)
        return HL_CUDA_ERROR;
    for (int i = 0; i < nimg; i++) {
        const int c = std::max(0, std::min(h_counts[i], linesmax));
        counts[i] = c;
        if (c > 0)
            memcpy(lines + (size_t)i * K, b->h_res + sizeof(hl_line) * K * i,
                   sizeof(hl_line) * c);
    }
    return HL_NO_ERROR;
}

extern "C" int hl_autotune(hl_handle *h, const hl_image_desc *imgs, int nimg,
                           const int *thresholds, int linesmax,
                           hl_tune_entry *best, hl_tune_entry *tried,
                           int max_tried, int *ntried, void *stream)
{
    if (!h || !imgs || !best)
        return HL_NULL_POINTER;
    if (nimg <= 0)
        return HL_INVALID_DATA;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int maxr = hl_vote_max_rows();
    const int row_cand[] = {256, 512, 768, 1024, maxr};
    const int thr_cand[] = {512, 1024};
    const int K = std::max(linesmax, 1);
    hl_line *d_lines = nullptr;
    int *d_counts = nullptr;
    CK(cudaMalloc(&d_lines, sizeof(hl_line) * (size_t)K * nimg));
    if (cudaMalloc(&d_counts, sizeof(int) * nimg) != cudaSuccess) {
        cudaFree(d_lines);
        return HL_OUT_OF_MEM;
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int saved_rows = h->win_rows_override, saved_thr = h->threads_override;
    const int saved_graph = h->batch_graph;
    h->batch_graph = 0;
    hl_tune_entry bst = {0, 0, 3.0e38f};
    int n = 0, rc = HL_NO_ERROR;
    for (int ti = 0; ti < 2 && rc == HL_NO_ERROR; ti++) {
        for (int ri = 0; ri < 5 && rc == HL_NO_ERROR; ri++) {
            const int rows = std::min(row_cand[ri], maxr);
            if (ri < 4 && row_cand[ri] >= maxr)
                continue;   /* the last candidate covers it */
            h->win_rows_override = rows;
            h->threads_override = thr_cand[ti];
            /* warm-up (plans, allocates), then three timed calls */
            rc = batch_run(h, imgs, nimg, thresholds, K, d_lines, d_counts, s);
            if (rc != HL_NO_ERROR)
                break;
            cudaEventRecord(e0, s);
            for (int r = 0; r < 3 && rc == HL_NO_ERROR; r++)
                rc = batch_run(h, imgs, nimg, thresholds, K, d_lines, d_counts, s);
            cudaEventRecord(e1, s);
            if (cudaEventSynchronize(e1) != cudaSuccess) {
                rc = HL_CUDA_ERROR;
                break;
            }
            float ms = 0.0f;
            cudaEventElapsedTime(&ms, e0, e1);
            ms /= 3.0f;
            hl_tune_entry te = {rows, thr_cand[ti], ms};
            if (tried && n < max_tried)
                tried[n] = te;
            n++;
            if (ms < bst.ms)
                bst = te;
        }
    }
    int st = 0;
    if (rc == HL_NO_ERROR && batch_last_status(h, &st, s) == HL_NO_ERROR && st != 0)
        rc = HL_CUDA_ERROR;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(d_lines);
    cudaFree(d_counts);
    h->batch_graph = saved_graph;
    if (rc != HL_NO_ERROR || bst.threads == 0) {
        h->win_rows_override = saved_rows;
        h->threads_override = saved_thr;
        return rc != HL_NO_ERROR ? rc : HL_CUDA_ERROR;
    }
    h->win_rows_override = bst.window_rows;
    h->threads_override = bst.threads;
    *best = bst;
    if (ntried)
        *ntried = n;
    return HL_NO_ERROR;
}

/* ==================================================================== */
/* Proposal-guided batched path                                          */
/* ==================================================================== */

struct hl_prop_ws {
    __nv_bfloat16 *d_occ;          /* [n][256][256] */
    size_t cap_occ;
    unsigned char *d_tab;          /* pool descriptors + head geometries */
    size_t cap_tab;
    unsigned char *h_tab;
    size_t cap_htab;
    int4 *d_win;
    size_t cap_win;
    int *d_cnt;                    /* [0] windows [1] status [2..3] votes [4] cells */
    int *d_fb;                     /* per-image fall-back flags */
    size_t cap_fb;
    int *h_fb;                     /* pinned copy */
    size_t cap_hfb;
    hl_line *d_fb_lines;           /* plain results of the fall-back set */
    size_t cap_fb_lines;
    int *d_fb_counts;
    size_t cap_fb_counts;
    int *d_map;                    /* fall-back slot -> image */
    size_t cap_map;
};

static void prop_free(hl_handle *h)
{
    hl_prop_ws *p = h->pw;
    if (!p)
        return;
    void *dp[] = {p->d_occ, p->d_tab, p->d_win, p->d_cnt, p->d_fb, p->d_fb_lines,
                  p->d_fb_counts, p->d_map};
    for (void *q : dp)
        if (q)
            cudaFree(q);
    if (p->h_tab)
        cudaFreeHost(p->h_tab);
    if (p->h_fb)
        cudaFreeHost(p->h_fb);
    delete p;
    h->pw = nullptr;
}

/* copy fall-back results (slot q -> image map[q]) into the outputs */
__global__ void hl_scatter_results_kernel(const hl_line *src_lines,
                                          const int *src_counts, const int *map,
                                          int nmap, int K, hl_line *dst_lines,
                                          int *dst_counts)
{
    for (int q = blockIdx.x; q < nmap; q += gridDim.x) {
        const int i = map[q];
        if (i < 0)
            continue;
        for (int j = threadIdx.x; j < K; j += blockDim.x)
            dst_lines[(size_t)i * K + j] = src_lines[(size_t)q * K + j];
        if (threadIdx.x == 0)
            dst_counts[i] = src_counts[q];
    }
}

extern "C" int hl_proposal_batch(hl_handle *h, hl_net *net,
                                 const hl_image_desc *imgs, int nimg,
                                 const int *thresholds, int linesmax,
                                 const hl_proposal_opts *opts,
                                 hl_line *lines_dev, int *counts_dev,
                                 hl_proposal_stats *stats, void *stream)
{
    if (!h || !net || !imgs || !opts || !counts_dev)
        return HL_NULL_POINTER;
    if (linesmax > 0 && !lines_dev)
        return HL_NULL_POINTER;
    if (nimg <= 0 || nimg > 0xffff || !(opts->p_cut > 0.0f && opts->p_cut < 1.0f) ||
        opts->max_props < 0 || opts->dilate_rho < 0 || opts->dilate_theta < 0 ||
        opts->judge_every < 0 || opts->top_m < 0 || opts->top_m > 1024 ||
        !(opts->p_conf >= 0.0f && opts->p_conf < 1.0f))
        return HL_INVALID_DATA;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int K = std::max(linesmax, 0);
    if (!h->bw) {
        h->bw = new (std::nothrow) hl_batch_ws();
        if (!h->bw)
            return HL_OUT_OF_MEM;
    }
    if (!h->pw) {
        h->pw = new (std::nothrow) hl_prop_ws();
        if (!h->pw)
            return HL_OUT_OF_MEM;
    }
    hl_batch_ws *b = h->bw;
    hl_prop_ws *pw = h->pw;
    std::vector<hl_roi> rois((size_t)nimg);
    int rc;
    for (int i = 0; i < nimg; i++)
        if ((rc = roi_of(&imgs[i], &rois[i])) != HL_NO_ERROR)
            return rc;
    if ((rc = batch_plan(h, b, imgs, nimg, thresholds, K, lines_dev, counts_dev,
                         rois.data(), s)) != HL_NO_ERROR)
        return rc;
    h->last_batch = 1;

    /* pool descriptors and head geometries (host), window capacity */
    const size_t off_geo = align16(sizeof(hl_pool_img) * nimg);
    const size_t tab = off_geo + sizeof(hl_head_geom) * nimg;
    size_t max_bins = 1;
    int nk_fast = 0;
    std::vector<char> force((size_t)nimg, 0);
    if (!b->tab_event) {
        CK(cudaEventCreateWithFlags(&b->tab_read, cudaEventDisableTiming));
        b->tab_event = 1;
    }
    CK(cudaEventSynchronize(b->tab_read));   /* pw->h_tab reuse */
    if ((rc = grow_host(&pw->h_tab, &pw->cap_htab, tab)) != HL_NO_ERROR ||
        (rc = grow((void **)&pw->d_tab, &pw->cap_tab, tab)) != HL_NO_ERROR ||
        (rc = grow((void **)&pw->d_occ, &pw->cap_occ,
                   sizeof(__nv_bfloat16) * 256 * 256 * (size_t)nimg)) != HL_NO_ERROR ||
        (rc = grow((void **)&pw->d_fb, &pw->cap_fb, sizeof(int) * nimg)) != HL_NO_ERROR ||
        (rc = grow_host((unsigned char **)&pw->h_fb, &pw->cap_hfb, sizeof(int) * nimg)) !=
            HL_NO_ERROR)
        return rc;
    if (!pw->d_cnt)
        CK(cudaMalloc(&pw->d_cnt, 8 * sizeof(int)));
    hl_pool_img *pi = reinterpret_cast<hl_pool_img *>(pw->h_tab);
    hl_head_geom *hg = reinterpret_cast<hl_head_geom *>(pw->h_tab + off_geo);
    for (int i = 0; i < nimg; i++) {
        const int w = rois[i].w, hh = rois[i].h;
        const int f = std::max(1, (std::max(w, hh) + 255) / 256);
        pi[i].base = rois[i].base;
        pi[i].pitch = rois[i].pitch;
        pi[i].w = w;
        pi[i].h = hh;
        pi[i].factor = f;
        pi[i].pad = 0;
        hg[i].cell = (float)(4 * f);
        hg[i].rho_min = (float)b->rho_min[i];
        hg[i].inv_rw = (float)HL_COARSE_R / (float)b->R[i];
        hg[i].qh = ((hh + f - 1) / f + 3) / 4;
        hg[i].qw = ((w + f - 1) / f + 3) / 4;
        hg[i].pad = 0;
        const int nk = (h->T + HL_COARSE_T - 1) / HL_COARSE_T + 2;
        const int nj = HL_WIN_RUN * ((b->R[i] + HL_COARSE_R - 1) / HL_COARSE_R) + 2;
        /* columns of nj rows plus a dump row; the branch-free vote for at
         * most 6 or 10 thetas writes that many columns */
        nk_fast = nk <= 6 ? 6 : (nk <= 10 ? 10 : 0);
        max_bins = std::max(max_bins, (size_t)std::max(nk, nk_fast) * (size_t)(nj + 1));
        const int ntiles = ((w + HL_TILE_W - 1) / HL_TILE_W) * ((hh + HL_TILE_H - 1) / HL_TILE_H);
        if (ntiles > HL_WIN_MAXTILES)
            force[i] = 1;
    }
    if (max_bins * sizeof(int) > 200u * 1024u)
        return HL_OP_OVERFLOW;
    const int cap_win = nimg * (std::max(1, opts->max_props) + std::max(0, opts->top_m) + 64) *
                        (2 * opts->dilate_rho + 1) * (2 * opts->dilate_theta + 1);
    if ((rc = grow((void **)&pw->d_win, &pw->cap_win, sizeof(int4) * (size_t)cap_win)) !=
        HL_NO_ERROR)
        return rc;

    /* device work: compaction, pooling, network, selection, windows, finalize */
    unsigned char *dt = b->d_tab;
    CK(cudaMemsetAsync(pw->d_cnt, 0, 8 * sizeof(int), s));
    CK(cudaMemcpyAsync(pw->d_tab, pw->h_tab, tab, cudaMemcpyHostToDevice, s));
    if ((rc = batch_enqueue_compact(h, b, nimg, s)) != HL_NO_ERROR)
        return rc;
    CK(hl_launch_pool(reinterpret_cast<const hl_pool_img *>(pw->d_tab), nimg, 256, pw->d_occ, s));
    const float *logits = nullptr;
    if ((rc = hl_net_run(net, pw->d_occ,
                         reinterpret_cast<const hl_head_geom *>(pw->d_tab + off_geo), nimg,
                         &logits, s)) != HL_NO_ERROR)
        return rc;
    hl_select_args sa;
    memset(&sa, 0, sizeof(sa));
    sa.logits = logits;
    sa.zcut = logf(opts->p_cut / (1.0f - opts->p_cut));
    sa.max_props = opts->max_props;
    sa.top_m = opts->top_m;
    sa.dil_t = opts->dilate_theta;
    sa.dil_r = opts->dilate_rho;
    sa.force_fallback = 0;
    sa.nms = opts->nms ? 1 : 0;
    sa.use_conf = opts->p_conf > 0.0f ? 1 : 0;
    sa.zconf = sa.use_conf ? logf(opts->p_conf / (1.0f - opts->p_conf)) : 0.0f;
    sa.fallback = pw->d_fb;
    sa.win = pw->d_win;
    sa.nwin = pw->d_cnt + 0;
    sa.ncells = pw->d_cnt + 4;
    sa.cap = cap_win;
    sa.status = pw->d_cnt + 1;
    CK(hl_launch_select(&sa, nimg, s));
    hl_window_args wa;
    memset(&wa, 0, sizeof(wa));
    wa.win = pw->d_win;
    wa.nwin = pw->d_cnt + 0;
    wa.cap = cap_win;
    wa.vimgs = reinterpret_cast<const hl_vote_img *>(dt + b->off_vimg);
    wa.pimgs = reinterpret_cast<const hl_peak_img *>(dt + b->off_pimg);
    wa.cosv = h->d_cos;
    wa.sinv = h->d_sin;
    wa.T = h->T;
    wa.irho = (float)(1.0 / h->p.derho);
    wa.votes = stats ? reinterpret_cast<unsigned long long *>(pw->d_cnt + 2) : nullptr;
    wa.status = pw->d_cnt + 1;
    wa.nk_fast = nk_fast;
    CK(hl_launch_window_vote(&wa, (int)max_bins, std::max(1, h->sms) * 6, s));
    if ((rc = batch_enqueue_finalize(h, b, nimg, K, false, s)) != HL_NO_ERROR)
        return rc;
    CK(cudaEventRecord(b->tab_read, s));

    /* fall-back and judged images run the plain method on the points that are
     * there already (32 x 2048 x 2048, 21 of them: 757 us, 792 with their own
     * compaction) */
    int st_host[5] = {0, 0, 0, 0, 0};
    CK(cudaMemcpyAsync(pw->h_fb, pw->d_fb, sizeof(int) * nimg, cudaMemcpyDeviceToHost, s));
    CK(cudaMemcpyAsync(st_host, pw->d_cnt, sizeof(st_host), cudaMemcpyDeviceToHost, s));
    int nst = 0;
    if ((rc = hl_net_status(net, &nst, s)) != HL_NO_ERROR)
        return rc;
    CK(cudaStreamSynchronize(s));
    if (st_host[1] != 0 || nst != 0)
        return HL_CUDA_ERROR;
    std::vector<int> sub, sub_fb;    /* images to run plain; is it a fall-back */
    for (int i = 0; i < nimg; i++) {
        const bool fb = pw->h_fb[i] != 0 || force[i];
        const bool judge = !fb && opts->judge_every > 0 && i % opts->judge_every == 0;
        if (fb || judge) {
            sub.push_back(i);
            sub_fb.push_back(fb ? 1 : 0);
        }
    }
    int n_fb = 0, judged = 0, jl = 0, jf = 0, n_conf = 0;
    for (int i = 0; i < nimg; i++)
        n_conf += pw->h_fb[i] == 2;
    if (!sub.empty()) {
        const int ns = (int)sub.size();
        std::vector<hl_image_desc> sd((size_t)ns);
        std::vector<int> sthr((size_t)ns);
        for (int q = 0; q < ns; q++) {
            sd[q] = imgs[sub[q]];
            sthr[q] = thresholds ? thresholds[sub[q]] : h->p.threshold;
        }
        const size_t KK = (size_t)std::max(K, 1);
        if ((rc = grow((void **)&pw->d_fb_lines, &pw->cap_fb_lines,
                       sizeof(hl_line) * KK * ns)) != HL_NO_ERROR ||
            (rc = grow((void **)&pw->d_fb_counts, &pw->cap_fb_counts, sizeof(int) * ns)) !=
                HL_NO_ERROR ||
            (rc = grow((void **)&pw->d_map, &pw->cap_map, sizeof(int) * ns)) != HL_NO_ERROR)
            return rc;
        if ((rc = batch_run_ws(h, &h->bw_fb, sd.data(), ns, sthr.data(), K, pw->d_fb_lines,
                               pw->d_fb_counts, s, h->bw, sub.data())) != HL_NO_ERROR)
            return rc;
        h->last_batch = 1;
        std::vector<int> map((size_t)ns, -1);
        for (int q = 0; q < ns; q++)
            if (sub_fb[q]) {
                map[q] = sub[q];
                n_fb++;
            }
        CK(cudaMemcpyAsync(pw->d_map, map.data(), sizeof(int) * ns, cudaMemcpyHostToDevice, s));
        if (n_fb > 0) {
            hl_scatter_results_kernel<<<std::min(ns, 1024), 128, 0, s>>>(
                pw->d_fb_lines, pw->d_fb_counts, pw->d_map, ns, K, lines_dev, counts_dev);
            CK(cudaGetLastError());
        }
        int fst = 0;
        CK(cudaMemcpyAsync(&fst, h->bw_fb->d_cnt + 2, sizeof(int), cudaMemcpyDeviceToHost, s));
        /* recall of the judged images: plain lines found by the proposals */
        std::vector<hl_line> pl, pp;
        std::vector<int> pc, qc;
        const int nj = ns - n_fb;
        if (nj > 0 && K > 0) {
            pl.resize(KK * ns);
            pc.resize(ns);
            pp.resize(KK * nimg);
            qc.resize(nimg);
            CK(cudaMemcpyAsync(pl.data(), pw->d_fb_lines, sizeof(hl_line) * KK * ns,
                               cudaMemcpyDeviceToHost, s));
            CK(cudaMemcpyAsync(pc.data(), pw->d_fb_counts, sizeof(int) * ns,
                               cudaMemcpyDeviceToHost, s));
            for (int q = 0; q < ns; q++) {
                if (sub_fb[q])
                    continue;
                const int i = sub[q];
                CK(cudaMemcpyAsync(pp.data() + KK * i, lines_dev + (size_t)i * K,
                                   sizeof(hl_line) * K, cudaMemcpyDeviceToHost, s));
                CK(cudaMemcpyAsync(qc.data() + i, counts_dev + i, sizeof(int),
                                   cudaMemcpyDeviceToHost, s));
            }
        }
        CK(cudaStreamSynchronize(s));
        if (batch_status(h->bw_fb, fst) != 0)
            return HL_CUDA_ERROR;
        if (nj > 0 && K > 0) {
            for (int q = 0; q < ns; q++) {
                if (sub_fb[q])
                    continue;
                const int i = sub[q];
                judged++;
                const int np = std::min(pc[q], K), nq = std::min(qc[i], K);
                jl += np;
                for (int a = 0; a < np; a++) {
                    const hl_line &L = pl[KK * q + a];
                    for (int c = 0; c < nq; c++) {
                        const hl_line &M = pp[KK * i + c];
                        if (M.angle == L.angle && M.distance == L.distance &&
                            M.votes == L.votes) {
                            jf++;
                            break;
                        }
                    }
                }
            }
        }
    }
    if (stats) {
        stats->fallback = n_fb;
        stats->windows = std::min(st_host[0], cap_win);
        stats->judged = judged;
        stats->judged_lines = jl;
        stats->judged_found = jf;
        stats->fallback_conf = n_conf;
        unsigned long long v = 0;
        memcpy(&v, &st_host[2], sizeof(v));
        stats->votes = (long long)v;
        stats->cells = st_host[4];
        stats->pad = 0;
    }
    return HL_NO_ERROR;
}

/* ---- HoughCircle (include/hl_circle.h) ---------------------------------- */

static int circle_prepare(hl_handle *h, const hl_image_desc *img, const hl_circle_params *p,
                          hl_roi *roi, hl_geom *g)
{
    if (!h || !img || !p)
        return HL_NULL_POINTER;
    if (p->radius_min < 0 || p->radius_max < p->radius_min || p->radius_max >= 65536 ||
        p->threshold < 0 || !(p->dist_thres == p->dist_thres))
        return HL_INVALID_DATA;
    int rc = roi_of(img, roi);
    if (rc != HL_NO_ERROR)
        return rc;
    return hl_geometry(h, roi->w, roi->h, g);
}

/* radii of [radius_min, radius_max] that are counted on bit planes: the smallest */
static int circle_dense(const hl_circle_params *p)
{
    return std::max(0, std::min(p->radius_max, HL_CIRCLE_DENSE_R) - p->radius_min + 1);
}

/* the table of circle offsets, made once a handle and waited for, so that later
 * calls may come on other streams; sets the kernel's pointers */
static int circle_table(hl_handle *h, hl_circle_bits_args *ba, cudaStream_t s)
{
    if (!h->d_ctab) {
        int *d = nullptr;
        CK(cudaMalloc(&d, hl_circle_table_bytes()));
        cudaError_t e = hl_launch_circle_table(d, s);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            cudaFree(d);
            return map_err(e);
        }
        h->d_ctab = d;
    }
    ba->table = h->d_ctab;
    ba->count = h->d_ctab + hl_circle_table_bytes() / sizeof(int) - (HL_CIRCLE_DENSE_R + 1);
    return HL_NO_ERROR;
}

static long long circle_bits_blocks(const hl_circle_bits_img &b)
{
    return ((long long)b.pitch * b.h + 255) / 256;
}

/* The smaller radii on bit planes of the edge map; the larger ones by the
 * compaction and one tile-kernel launch: the accumulator written to acc
 * ([nr][h][w]) when it is given, the local maxima appended to the handle's
 * candidate keys when peaks is set */
static int circle_run(hl_handle *h, const hl_roi &roi, const hl_geom &g,
                      const hl_circle_params *p, int32_t *acc, bool peaks, cudaStream_t s)
{
    const int nr = p->radius_max - p->radius_min + 1;
    hl_circle_tile_args ta;
    memset(&ta, 0, sizeof(ta));
    ta.ntx = (roi.w + HL_CIRCLE_TW - 1) / HL_CIRCLE_TW;
    ta.nty = (roi.h + HL_CIRCLE_TH - 1) / HL_CIRCLE_TH;
    if ((long long)ta.ntx * ta.nty * nr > 0x7fffffffLL)
        return HL_OP_OVERFLOW;   /* more CTAs than one launch takes */
    int rc;
    const int nd = circle_dense(p);
    if (nd > 0) {
        hl_circle_bits_args ba;
        memset(&ba, 0, sizeof(ba));
        hl_circle_bits_img &b = ba.img0;
        b.roi = roi;
        b.w = roi.w;
        b.h = roi.h;
        hl_circle_bits_tiles(&b);
        if ((rc = circle_table(h, &ba, s)) != HL_NO_ERROR ||
            (rc = grow((void **)&h->d_cbits, &h->cap_cbits,
                       sizeof(uint32_t) * (size_t)b.pitch * (size_t)b.h)) != HL_NO_ERROR)
            return rc;
        b.bits = h->d_cbits;
        ba.nimg = 1;
        ba.rmin = p->radius_min;
        ba.nr = nd;
        ba.acc = acc;
        ba.threshold = p->threshold;
        if (peaks) {
            ba.keys = h->d_ckeys;
            ba.ncand = h->d_ccnt;
            ba.cap = HL_CIRCLE_MAXCAND;
            ba.status = h->d_ccnt + 1;
        }
        CK(hl_launch_edge_bits(nullptr, &b, 1, circle_bits_blocks(b), s));
        CK(hl_launch_circle_bits(&ba, (long long)b.ntx * b.nty * nd, b.twu, s));
    }
    if (nd == nr)
        return HL_NO_ERROR;
    if ((rc = ensure_image(h, g, roi.w, roi.h, s)) != HL_NO_ERROR ||
        (rc = launch_compaction(h, roi, g, s)) != HL_NO_ERROR)
        return rc;
    ta.nz = nr - nd;
    ta.pts = reinterpret_cast<const float2 *>(h->d_pts);
    ta.tile_off = h->d_tile_off;
    ta.ctiles_x = g.tiles_x;
    ta.ctiles_y = g.tiles_y;
    ta.w = roi.w;
    ta.h = roi.h;
    ta.rmin = p->radius_min;
    ta.nr = nr;
    ta.acc = acc;
    ta.threshold = p->threshold;
    if (peaks) {
        ta.keys = h->d_ckeys;
        ta.ncand = h->d_ccnt;
        ta.cap = HL_CIRCLE_MAXCAND;
        ta.status = h->d_ccnt + 1;
    }
    CK(hl_launch_circle_tiles(&ta, s));
    return HL_NO_ERROR;
}

extern "C" int hl_circle_accumulator(hl_handle *h, const hl_image_desc *img,
                                     const hl_circle_params *p, int32_t *acc_dev,
                                     void *stream)
{
    if (!acc_dev)
        return HL_NULL_POINTER;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    hl_roi roi;
    hl_geom g;
    int rc = circle_prepare(h, img, p, &roi, &g);
    if (rc != HL_NO_ERROR)
        return rc;
    if ((rc = circle_run(h, roi, g, p, acc_dev, false, s)) != HL_NO_ERROR)
        return rc;
    /* the compaction's status word (a bounded wait that gave up) */
    int st = 0;
    CK(cudaMemcpyAsync(&st, h->d_counters + 1, sizeof(int), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (st != 0) {
        reset_counters(h, s);
        return HL_CUDA_ERROR;
    }
    return HL_NO_ERROR;
}

extern "C" int hl_circles(hl_handle *h, const hl_image_desc *img, const hl_circle_params *p,
                          int *circlemax, hl_circle *out, void *stream)
{
    if (!circlemax)
        return HL_NULL_POINTER;
    if (*circlemax > 0 && !out)
        return HL_NULL_POINTER;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    hl_roi roi;
    hl_geom g;
    int rc = circle_prepare(h, img, p, &roi, &g);
    if (rc != HL_NO_ERROR)
        return rc;
    const int nr = p->radius_max - p->radius_min + 1;
    const size_t cells = (size_t)nr * roi.w * roi.h;
    if (cells >= (size_t)0xffffffffu)
        return HL_OP_OVERFLOW;   /* the candidate key holds a 32-bit index */
    const int cm = std::max(*circlemax, 0);
    const size_t rbytes = sizeof(hl_result_hdr) + sizeof(hl_circle) * (size_t)std::max(cm, 1);
    if (!h->d_ckeys) {
        CK(cudaMalloc(&h->d_ckeys, sizeof(unsigned long long) * HL_CIRCLE_MAXCAND));
        CK(cudaMalloc(&h->d_ccnt, 2 * sizeof(int)));
        CK(cudaMemsetAsync(h->d_ccnt, 0, 2 * sizeof(int), s));
    }
    /* results: header + room for circlemax circles, pinned mirror */
    static const size_t kResCap = sizeof(hl_result_hdr) + sizeof(hl_circle) * 4096;
    if (rbytes > kResCap)
        return HL_INVALID_DATA;
    if (!h->d_cres) {
        CK(cudaMalloc(&h->d_cres, kResCap));
        CK(cudaMallocHost(&h->h_cres, kResCap + sizeof(int)));
    }
    if ((rc = circle_run(h, roi, g, p, nullptr, true, s)) != HL_NO_ERROR)
        return rc;
    hl_circle_final_args fa;
    fa.imgs = nullptr;
    fa.keys = h->d_ckeys;
    fa.ncand = h->d_ccnt;
    fa.w = roi.w;
    fa.h = roi.h;
    fa.rmin = p->radius_min;
    fa.dist_thres = p->dist_thres;
    fa.r_thres = p->r_thres;
    fa.circlemax = cm;
    fa.roi_x = img->roi_x1;
    fa.roi_y = img->roi_y1;
    fa.out = reinterpret_cast<hl_circle *>(h->d_cres + sizeof(hl_result_hdr));
    fa.hdr = reinterpret_cast<hl_result_hdr *>(h->d_cres);
    fa.status = h->d_ccnt + 1;
    CK(hl_launch_circle_final(&fa, 1, s));
    /* the results and the compaction's status word */
    int *cstat = reinterpret_cast<int *>(h->h_cres + kResCap);
    CK(cudaMemcpyAsync(h->h_cres, h->d_cres, rbytes, cudaMemcpyDeviceToHost, s));
    CK(cudaMemcpyAsync(cstat, h->d_counters + 1, sizeof(int), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    const hl_result_hdr *hdr = reinterpret_cast<const hl_result_hdr *>(h->h_cres);
    if (*cstat != 0) {
        reset_counters(h, s);
        return HL_CUDA_ERROR;
    }
    if (hdr->status != 0)
        return (hdr->status & HL_ST_CAND_OVERFLOW) ? HL_OP_OVERFLOW : HL_CUDA_ERROR;
    if (hdr->count > 0)
        memcpy(out, h->h_cres + sizeof(hl_result_hdr), sizeof(hl_circle) * (size_t)hdr->count);
    *circlemax = hdr->count;
    return HL_NO_ERROR;
}

/* ---- HoughCircle batches -------------------------------------------------- */

struct hl_cb_ws {
    float2 *d_pts;
    size_t cap_pts;
    int *d_toff;
    size_t cap_toff;
    unsigned long long *d_state;
    size_t cap_state;
    uint32_t *d_bits;
    size_t cap_bits;
    unsigned char *d_tab;
    size_t cap_tab;
    unsigned char *h_tab;
    size_t cap_htab;
    unsigned long long *d_keys;
    size_t cap_keys;
    int *d_cnt;
    size_t cap_cnt;
    unsigned char *d_res;
    size_t cap_res;
    unsigned char *h_res;
    size_t cap_hres;
};

static void circle_batch_free(hl_handle *h)
{
    hl_cb_ws *c = h->cb;
    if (!c)
        return;
    void *dp[] = {c->d_pts, c->d_toff, c->d_state, c->d_bits, c->d_tab, c->d_keys, c->d_cnt, c->d_res};
    for (void *q : dp)
        if (q)
            cudaFree(q);
    if (c->h_tab)
        cudaFreeHost(c->h_tab);
    if (c->h_res)
        cudaFreeHost(c->h_res);
    delete c;
    h->cb = nullptr;
}

/* Circles of many ROIs (of one image or several) in one pipeline: the edge maps
 * of every ROI and one bit-plane launch over their (tile, radius) CTAs, for the
 * larger radii one compaction over every ROI (the batch form of the compaction
 * kernel, each ROI its own point region and tile offsets) and one tile launch,
 * then one tail CTA per ROI, one copy of the results. */
extern "C" int hl_circles_batch(hl_handle *h, const hl_image_desc *imgs, int nimg,
                                const hl_circle_params *p, int circlemax, hl_circle *out,
                                int *counts, void *stream)
{
    if (!h || !p || !counts || (nimg > 0 && !imgs) || (nimg > 0 && circlemax > 0 && !out))
        return HL_NULL_POINTER;
    if (nimg < 0 || circlemax < 0 || circlemax > HL_CIRCLE_MAXCAND)
        return HL_INVALID_DATA;
    if (p->radius_min < 0 || p->radius_max < p->radius_min || p->radius_max >= 65536 ||
        p->threshold < 0 || !(p->dist_thres == p->dist_thres))
        return HL_INVALID_DATA;
    if (nimg == 0)
        return HL_NO_ERROR;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int nr = p->radius_max - p->radius_min + 1;
    std::vector<hl_roi> rois((size_t)nimg);
    std::vector<hl_geom> gs((size_t)nimg);
    std::vector<long long> pts_base((size_t)nimg);
    std::vector<int> tile_base((size_t)nimg), group_base((size_t)nimg), cta_base((size_t)nimg);
    std::vector<int> group_img;
    long long pts = 0, ctas = 0, blocks = 0, tiles = 0, groups = 0;
    const int nd = circle_dense(p);
    std::vector<hl_circle_bits_img> bi((size_t)nimg);
    long long bctas = 0, bblocks = 0;
    int twu_min = 8;
    for (int i = 0; i < nimg; i++) {
        int rc = roi_of(&imgs[i], &rois[i]);
        if (rc != HL_NO_ERROR)
            return rc;
        if ((rc = hl_geometry(h, rois[i].w, rois[i].h, &gs[i])) != HL_NO_ERROR)
            return rc;
        if ((size_t)nr * rois[i].w * rois[i].h >= (size_t)0xffffffffu)
            return HL_OP_OVERFLOW;   /* the candidate key holds a 32-bit index */
        const int nt = gs[i].tiles_x * gs[i].tiles_y;
        const int ng = (nt + HL_COMPACT_GROUP - 1) / HL_COMPACT_GROUP;
        tile_base[i] = (int)tiles;
        group_base[i] = (int)groups;
        for (int q = 0; q < ng; q++)
            group_img.push_back(i);
        tiles += nt + 1;   /* the ROI's tile offsets and its end */
        groups += ng;
        /* every pixel and one pad per tile, even so each region starts on
         * 16 bytes */
        pts_base[i] = pts;
        pts += ((long long)rois[i].w * rois[i].h + nt + 16 + 1) & ~1LL;
        const long long ntx = (rois[i].w + HL_CIRCLE_TW - 1) / HL_CIRCLE_TW;
        const long long nty = (rois[i].h + HL_CIRCLE_TH - 1) / HL_CIRCLE_TH;
        cta_base[i] = (int)std::min(ctas, (long long)0x7fffffff);
        ctas += ntx * nty * (nr - nd);
        blocks += ntx * nty * nr;
        bi[i].roi = rois[i];
        bi[i].w = rois[i].w;
        bi[i].h = rois[i].h;
        hl_circle_bits_tiles(&bi[i]);
        bi[i].cta_base = bctas;
        bctas += (long long)bi[i].ntx * bi[i].nty * nd;
        bi[i].blk_base = (int)std::min(bblocks, (long long)0x7fffffff);
        bblocks += circle_bits_blocks(bi[i]);
        twu_min = std::min(twu_min, bi[i].twu);
        if (blocks > 0x7fffffffLL || bblocks > 0x7fffffffLL || tiles > 0x7fffffffLL || groups > 0x7fffffffLL)
            return HL_OP_OVERFLOW;
    }
    if (!h->cb && !(h->cb = new (std::nothrow) hl_cb_ws()))
        return HL_OUT_OF_MEM;
    hl_cb_ws *c = h->cb;
    const size_t rstride =
        align16(sizeof(hl_result_hdr) + sizeof(hl_circle) * (size_t)std::max(circlemax, 1));
    const size_t off_cimg = 0;
    const size_t off_gimg = align16(sizeof(hl_compact_img) * (size_t)nimg);
    const size_t off_circ = align16(off_gimg + sizeof(int) * (size_t)groups);
    const size_t off_bits = align16(off_circ + sizeof(hl_circle_img) * (size_t)nimg);
    const size_t tab_bytes = align16(off_bits + sizeof(hl_circle_bits_img) * (size_t)nimg);
    const size_t ncnt = 4 + 2 * (size_t)nimg;   /* ticket, count, status, pad, per ROI */
    int rc;
    if ((nr > nd &&
         ((rc = grow((void **)&c->d_pts, &c->cap_pts, sizeof(float2) * (size_t)pts)) !=
              HL_NO_ERROR ||
          (rc = grow((void **)&c->d_toff, &c->cap_toff, sizeof(int) * (size_t)tiles)) !=
              HL_NO_ERROR ||
          (rc = grow((void **)&c->d_state, &c->cap_state,
                     sizeof(unsigned long long) * (size_t)(groups + 1))) != HL_NO_ERROR)) ||
        (rc = grow((void **)&c->d_bits, &c->cap_bits,
                   sizeof(uint32_t) * 256 * (size_t)bblocks)) != HL_NO_ERROR ||
        (rc = grow((void **)&c->d_tab, &c->cap_tab, tab_bytes)) != HL_NO_ERROR ||
        (rc = grow_host(&c->h_tab, &c->cap_htab, tab_bytes)) != HL_NO_ERROR ||
        (rc = grow((void **)&c->d_keys, &c->cap_keys,
                   sizeof(unsigned long long) * HL_CIRCLE_MAXCAND * (size_t)nimg)) != HL_NO_ERROR ||
        (rc = grow((void **)&c->d_cnt, &c->cap_cnt, sizeof(int) * ncnt)) != HL_NO_ERROR ||
        (rc = grow((void **)&c->d_res, &c->cap_res, rstride * (size_t)nimg)) != HL_NO_ERROR ||
        (rc = grow_host(&c->h_res, &c->cap_hres, rstride * (size_t)nimg + 16)) != HL_NO_ERROR)
        return rc;
    hl_compact_img *ci = reinterpret_cast<hl_compact_img *>(c->h_tab + off_cimg);
    hl_circle_img *im = reinterpret_cast<hl_circle_img *>(c->h_tab + off_circ);
    for (int i = 0; i < nimg; i++) {
        const hl_geom &g = gs[i];
        const int nt = g.tiles_x * g.tiles_y;
        ci[i].roi = rois[i];
        ci[i].tiles_x = g.tiles_x;
        ci[i].ntiles = nt;
        ci[i].tile_base = tile_base[i];
        ci[i].group_base = group_base[i];
        ci[i].ngroups = (nt + HL_COMPACT_GROUP - 1) / HL_COMPACT_GROUP;
        ci[i].pad = 0;
        ci[i].pts_base = pts_base[i];
        im[i].pts = c->d_pts + pts_base[i];
        im[i].tile_off = c->d_toff + tile_base[i];
        im[i].ctiles_x = g.tiles_x;
        im[i].ctiles_y = g.tiles_y;
        im[i].w = rois[i].w;
        im[i].h = rois[i].h;
        im[i].ntx = (rois[i].w + HL_CIRCLE_TW - 1) / HL_CIRCLE_TW;
        im[i].nty = (rois[i].h + HL_CIRCLE_TH - 1) / HL_CIRCLE_TH;
        im[i].roi_x = imgs[i].roi_x1;
        im[i].roi_y = imgs[i].roi_y1;
        im[i].cta_base = cta_base[i];
        im[i].pad = 0;
        im[i].keys = c->d_keys + (size_t)HL_CIRCLE_MAXCAND * i;
        im[i].ncand = c->d_cnt + 4 + 2 * i;
        im[i].hdr = reinterpret_cast<hl_result_hdr *>(c->d_res + rstride * i);
        im[i].out = reinterpret_cast<hl_circle *>(c->d_res + rstride * i + sizeof(hl_result_hdr));
        bi[i].bits = c->d_bits + 256 * (size_t)bi[i].blk_base;
        bi[i].keys = im[i].keys;
        bi[i].ncand = im[i].ncand;
    }
    memcpy(c->h_tab + off_bits, bi.data(), sizeof(hl_circle_bits_img) * (size_t)nimg);
    memcpy(c->h_tab + off_gimg, group_img.data(), sizeof(int) * group_img.size());
    unsigned char *dt = c->d_tab;
    CK(cudaMemsetAsync(c->d_cnt, 0, sizeof(int) * ncnt, s));
    CK(cudaMemcpyAsync(dt, c->h_tab, tab_bytes, cudaMemcpyHostToDevice, s));
    if (nd > 0) {
        hl_circle_bits_args ba;
        memset(&ba, 0, sizeof(ba));
        if ((rc = circle_table(h, &ba, s)) != HL_NO_ERROR)
            return rc;
        ba.imgs = reinterpret_cast<const hl_circle_bits_img *>(dt + off_bits);
        ba.nimg = nimg;
        ba.rmin = p->radius_min;
        ba.nr = nd;
        ba.threshold = p->threshold;
        ba.keys = c->d_keys;   /* each image's own: see imgs */
        ba.cap = HL_CIRCLE_MAXCAND;
        CK(hl_launch_edge_bits(ba.imgs, &ba.img0, nimg, bblocks, s));
        CK(hl_launch_circle_bits(&ba, bctas, twu_min, s));
    }
    if (nr > nd) {
        CK(cudaMemsetAsync(c->d_state, 0, sizeof(unsigned long long) * (size_t)(groups + 1), s));
        hl_compact_args ca;
        memset(&ca, 0, sizeof(ca));
        ca.imgs = reinterpret_cast<const hl_compact_img *>(dt + off_cimg);
        ca.group_img = reinterpret_cast<const int *>(dt + off_gimg);
        ca.nimg = nimg;
        ca.ngroups = (int)groups;
        ca.tile_state = c->d_state;
        ca.ticket = reinterpret_cast<unsigned *>(c->d_cnt + 0);
        ca.ticket_base = 0;
        ca.epoch = 1;
        ca.pts = nullptr;
        ca.pts_f2 = c->d_pts;
        ca.tile_off = c->d_toff;
        ca.count = c->d_cnt + 1;
        ca.status = c->d_cnt + 2;
        CK(hl_launch_compact(&ca, s));
        hl_circle_tile_args ta;
        memset(&ta, 0, sizeof(ta));
        ta.imgs = reinterpret_cast<const hl_circle_img *>(dt + off_circ);
        ta.nimg = nimg;
        ta.nctas = (int)ctas;
        ta.rmin = p->radius_min;
        ta.nr = nr;
        ta.nz = nr - nd;
        ta.acc = nullptr;
        ta.threshold = p->threshold;
        ta.cap = HL_CIRCLE_MAXCAND;
        CK(hl_launch_circle_tiles(&ta, s));
    }
    hl_circle_final_args fa;
    memset(&fa, 0, sizeof(fa));
    fa.imgs = reinterpret_cast<const hl_circle_img *>(dt + off_circ);
    fa.rmin = p->radius_min;
    fa.dist_thres = p->dist_thres;
    fa.r_thres = p->r_thres;
    fa.circlemax = circlemax;
    CK(hl_launch_circle_final(&fa, nimg, s));
    int *cstat = reinterpret_cast<int *>(c->h_res + rstride * (size_t)nimg);
    CK(cudaMemcpyAsync(c->h_res, c->d_res, rstride * (size_t)nimg, cudaMemcpyDeviceToHost, s));
    CK(cudaMemcpyAsync(cstat, c->d_cnt + 2, sizeof(int), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (*cstat != 0)
        return HL_CUDA_ERROR;
    rc = HL_NO_ERROR;
    for (int i = 0; i < nimg; i++) {
        const hl_result_hdr *hdr =
            reinterpret_cast<const hl_result_hdr *>(c->h_res + rstride * (size_t)i);
        if (hdr->status != 0) {
            counts[i] = 0;
            if (rc == HL_NO_ERROR)
                rc = (hdr->status & HL_ST_CAND_OVERFLOW) ? HL_OP_OVERFLOW : HL_CUDA_ERROR;
            continue;
        }
        counts[i] = hdr->count;
        if (hdr->count > 0)
            memcpy(out + (size_t)circlemax * i, c->h_res + rstride * (size_t)i + sizeof(hl_result_hdr),
                   sizeof(hl_circle) * (size_t)hdr->count);
    }
    return rc;
}

