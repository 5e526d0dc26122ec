/*
 * hl_cnn.h -- kernel argument blocks and launchers of the proposal network
 * (not part of the C ABI).
 */
#ifndef HL_CNN_H
#define HL_CNN_H

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

/* The gradients are summed into this many copies of the flat parameters (a
 * CTA adds to copy blockIdx % HL_GRAD_COPIES), which the update kernel adds up:
 * hundreds of CTAs reducing into one address otherwise queue at its L2 line. */
#define HL_GRAD_COPIES 8

/* 3x3 convolution, padding 1: x [B][H][W][cin] -> y [B][Ho][Wo][cout] */
typedef struct hl_conv_args {
    const __nv_bfloat16 *x;
    const __nv_bfloat16 *w;   /* [cout][kreal], kreal = 9 * cin */
    const float *bias;        /* [cout] or NULL */
    __nv_bfloat16 *y;         /* bf16 NHWC with 32 channels ... */
    float *y_f32;             /* ... or f32 [B][Ho][Wo] when cout == 1 */
    int B, H, W, Ho, Wo;
    int cin, cout, kreal;
    int stride;
    int relu;
    /* w and bias were written before the launch preceding this one on its
     * stream began: they may be read while that one still runs */
    int w_ready;
    int *status;
    /* an input gradient of the network (NULL: none): masked by the ReLU output
     * mask (the layout of y), its sums over the pixels added to db [cout] of a
     * gradient copy (db_stride floats apart) */
    const __nv_bfloat16 *mask;
    float *db;
    int db_stride;
} hl_conv_args;

/* mode 0: convolution; mode 1: input gradient of a stride-2 convolution
 * (x = dy, w = the transposed weights [cin][9 * cout], Ho x Wo = the input
 * size of the forward convolution) */
cudaError_t hl_launch_conv3x3(const hl_conv_args *a, int mode, cudaStream_t s);

/* Weight gradient of a 3x3 convolution (padding 1): dw [cout][9 * cin] of a
 * gradient copy (dw_stride floats apart) +=.
 * x as in the forward pass; dy bf16 [P][32] (cout = 32), or dy NULL and
 * dy_f32 [P] (cout = 1, cin = 32, stride 1). */
typedef struct hl_dw_args {
    const __nv_bfloat16 *x;
    const __nv_bfloat16 *dy;
    const float *dy_f32;
    float *dw;
    int dw_stride;
    int B, H, W, Ho, Wo;
    int cin;
    int stride;
    int *status;
} hl_dw_args;
cudaError_t hl_launch_conv_dw(const hl_dw_args *a, cudaStream_t s);

/* Average pooling of 0/255 images into side x side occupancy maps. */
typedef struct hl_pool_img {
    const uint8_t *base;   /* ROI origin */
    long pitch;
    int w, h;
    int factor;            /* pooled cell = factor x factor pixels */
    int pad;
} hl_pool_img;
cudaError_t hl_launch_pool(const hl_pool_img *imgs, int nimg, int side,
                           __nv_bfloat16 *out, cudaStream_t s);

/* The fixed coarse Hough head: HL_HEAD_T angles (cell centres of
 * 180 / HL_HEAD_T degrees) x HL_HEAD_R rho bins over the image's rho range. */
#define HL_HEAD_T 90
#define HL_HEAD_R 128
typedef struct hl_head_geom {
    float cell;      /* evidence cell size in image pixels */
    float rho_min;   /* the image's rho range start */
    float inv_rw;    /* coarse bins per rho unit: 128 / R */
    int qh, qw;      /* evidence cells covering the ROI */
    int pad;
} hl_head_geom;
/* e: [nimg][64][64] evidence; hsum may be NULL (no training) */
cudaError_t hl_launch_head_fwd(const float *e, const hl_head_geom *geo,
                               int nimg, const float *ab, float *hsum,
                               float *logits, cudaStream_t s);
cudaError_t hl_launch_head_bwd(const float *dz, int ev, const hl_head_geom *geo,
                               int nimg, const float *ab, float *de, __nv_bfloat16 *de_b,
                               float *db, int db_stride, cudaStream_t s);
cudaError_t hl_launch_bce(const float *z, const float *y, const float *hsum,
                          long long n, float wpos, float *dz, float *dab,
                          float *loss, int stride, cudaStream_t s);
/* The optimiser step and the bf16 weight copies of every layer. */
#define HL_NET_LAYERS 6
typedef struct hl_update_layer {
    int off, cout, cin;       /* its weights in the flat parameters */
    int flip;                 /* wb: taps mirrored (stride 1) */
    __nv_bfloat16 *wf, *wb;   /* wb NULL: no backward copy */
} hl_update_layer;
typedef struct hl_update_args {
    float *w;
    float *g;                 /* [n] and the loss: the copies' sums (gsum) */
    float *m, *v;
    const float *gpart;       /* HL_GRAD_COPIES x gstride: [n] and the loss each */
    int gstride, gsum;
    int n;
    float lr, clip;           /* lr = 0: only the copies */
    float c1, c2;             /* bias corrections (set by the launcher) */
    int nlayers;
    hl_update_layer layer[HL_NET_LAYERS];
} hl_update_args;
cudaError_t hl_launch_update(hl_update_args *a, int step, cudaStream_t s);

struct hl_net;
/* the network's forward pass on device-resident geometry (hl_proposal.cpp);
 * *logits points into the network's own buffer */
int hl_net_run(struct hl_net *n, const __nv_bfloat16 *occ,
               const hl_head_geom *geo_dev, int B, const float **logits,
               cudaStream_t s);
/* stream-ordered copy of the network's status word into *st (pinned) */
int hl_net_status(struct hl_net *n, int *st, cudaStream_t s);

#endif
