/*
 * hl_proposal.cpp -- the C ABI of the proposal network: single-layer entry
 * points (used by the parity tests), the network object (forward, training
 * step with the project's own backward kernels and Adam) and the
 * proposal-guided HoughLine pipeline.
 */
#include <cuda_runtime.h>

#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <new>
#include <vector>

#include "hl_cnn.h"
#include "hl_internal.h"
#include "hl_proposal.h"

static int cnn_err(cudaError_t e)
{
    if (e == cudaSuccess)
        return HL_NO_ERROR;
    cudaGetLastError();   /* reported once: see map_err in hl_api.cpp */
    return e == cudaErrorMemoryAllocation ? HL_OUT_OF_MEM : HL_CUDA_ERROR;
}

#define CKN(call)                                 \
    do {                                          \
        cudaError_t e__ = (call);                 \
        if (e__ != cudaSuccess)                   \
            return cnn_err(e__);                  \
    } while (0)

extern "C" int hl_cnn_conv3x3(const void *x, const void *w, const float *bias,
                              void *y, float *y_f32, int B, int H, int W,
                              int cin, int cout, int stride, int relu,
                              int mode, int *status_dev, void *stream)
{
    if (!x || !w || (!y && !y_f32) || !status_dev)
        return HL_NULL_POINTER;
    if (B <= 0 || H <= 0 || W <= 0 || (cin != 1 && cin != 32) || cout < 1 ||
        cout > 32 || (stride != 1 && stride != 2) || (mode != 0 && mode != 1))
        return HL_INVALID_DATA;
    if ((y_f32 && cout != 1) || (mode == 1 && (stride != 2 || cin != 32)))
        return HL_INVALID_DATA;
    hl_conv_args a;
    memset(&a, 0, sizeof(a));
    a.x = static_cast<const __nv_bfloat16 *>(x);
    a.w = static_cast<const __nv_bfloat16 *>(w);
    a.bias = bias;
    a.y = static_cast<__nv_bfloat16 *>(y);
    a.y_f32 = y_f32;
    a.B = B;
    a.H = H;
    a.W = W;
    if (mode == 0) {
        a.Ho = (H - 1) / stride + 1;
        a.Wo = (W - 1) / stride + 1;
    } else {   /* x-gradient of a stride-2 conv whose input was 2H x 2W */
        a.Ho = 2 * H;
        a.Wo = 2 * W;
    }
    a.cin = cin;
    a.cout = cout;
    a.kreal = 9 * cin;
    a.stride = stride;
    a.relu = relu;
    a.status = status_dev;
    CKN(hl_launch_conv3x3(&a, mode, reinterpret_cast<cudaStream_t>(stream)));
    return HL_NO_ERROR;
}

/* ==================================================================== */
/* The network                                                           */
/* ==================================================================== */

/* Layers: (cin, cout, stride, relu); input 256 x 256 x 1, evidence 64 x 64. */
#define NET_LAYERS HL_NET_LAYERS
static const int L_CIN[NET_LAYERS] = {1, 32, 32, 32, 32, 32};
static const int L_COUT[NET_LAYERS] = {32, 32, 32, 32, 32, 1};
static const int L_STRIDE[NET_LAYERS] = {2, 2, 1, 1, 1, 1};
static const int L_RELU[NET_LAYERS] = {1, 1, 1, 1, 1, 0};
#define NET_IN 256
#define NET_EV 64

/* flat FP32 parameter offsets: per layer W [cout][9 cin] then b [cout]; then
 * the head's alpha, beta */
static int w_off(int l)
{
    int o = 0;
    for (int i = 0; i < l; i++)
        o += L_COUT[i] * 9 * L_CIN[i] + L_COUT[i];
    return o;
}
static int b_off(int l) { return w_off(l) + L_COUT[l] * 9 * L_CIN[l]; }
static int ab_off(void) { return w_off(NET_LAYERS); }
static int n_params(void) { return ab_off() + 2; }
/* floats of a gradient copy: the parameters and the loss, whole 128-byte lines */
static int g_stride(void) { return (n_params() + 1 + 31) / 32 * 32; }

/* side of layer l's input and output */
static int l_in_side(int l) { return l == 0 ? NET_IN : (l == 1 ? NET_IN / 2 : NET_EV); }
static int l_out_side(int l) { return l == 0 ? NET_IN / 2 : NET_EV; }

struct hl_net {
    int B;                             /* capacity (images) */
    float *w, *g, *m, *v;              /* FP32 master weights, grads, Adam */
    float *gpart;                      /* gradient copies, each [np] and the loss */
    __nv_bfloat16 *wf[NET_LAYERS];     /* forward bf16 weights */
    __nv_bfloat16 *wb[NET_LAYERS];     /* backward layouts (l >= 1) */
    __nv_bfloat16 *act[NET_LAYERS];    /* outputs of layers 0..4 (bf16) */
    float *ev;                         /* layer 5 output, [B][64][64] */
    float *hsum, *logits, *dz;         /* [B][90][128] */
    float *de;                         /* [B][64][64] */
    __nv_bfloat16 *de_b;
    __nv_bfloat16 *gx, *gx2;           /* masked input gradients (bf16, 32 ch) */
    float *loss;                       /* after the gradients */
    int *status;                       /* after the loss: read back with it */
    hl_head_geom *geo;                 /* [B] */
    int step;
};

static void net_free_bufs(hl_net *n)
{
    void *p[] = {n->ev, n->hsum, n->logits, n->dz, n->de, n->de_b, n->gx, n->gx2, n->geo};
    for (void *q : p)
        if (q)
            cudaFree(q);
    for (int l = 0; l < NET_LAYERS; l++)
        if (n->act[l])
            cudaFree(n->act[l]);
    n->ev = n->hsum = n->logits = n->dz = n->de = nullptr;
    n->de_b = n->gx = n->gx2 = nullptr;
    n->geo = nullptr;
    for (int l = 0; l < NET_LAYERS; l++)
        n->act[l] = nullptr;
    n->B = 0;
}

static int net_reserve(hl_net *n, int B)
{
    if (B <= n->B)
        return HL_NO_ERROR;
    net_free_bufs(n);
    const size_t s128 = (size_t)B * 128 * 128, s64 = (size_t)B * 64 * 64;
    const size_t cells = (size_t)B * HL_HEAD_T * HL_HEAD_R;
    CKN(cudaMalloc(&n->act[0], s128 * 32 * sizeof(__nv_bfloat16)));
    for (int l = 1; l < 5; l++)
        CKN(cudaMalloc(&n->act[l], s64 * 32 * sizeof(__nv_bfloat16)));
    CKN(cudaMalloc(&n->ev, s64 * sizeof(float)));
    CKN(cudaMalloc(&n->hsum, cells * sizeof(float)));
    CKN(cudaMalloc(&n->logits, cells * sizeof(float)));
    CKN(cudaMalloc(&n->dz, cells * sizeof(float)));
    CKN(cudaMalloc(&n->de, s64 * sizeof(float)));
    CKN(cudaMalloc(&n->de_b, s64 * sizeof(__nv_bfloat16)));
    CKN(cudaMalloc(&n->gx, s128 * 32 * sizeof(__nv_bfloat16)));
    CKN(cudaMalloc(&n->gx2, s128 * 32 * sizeof(__nv_bfloat16)));
    CKN(cudaMalloc(&n->geo, (size_t)B * sizeof(hl_head_geom)));
    n->B = B;
    return HL_NO_ERROR;
}

/* one optimiser step (lr > 0) and the bf16 copies of the master weights in
 * every layout the passes use */
static int net_update(hl_net *n, float lr, bool gsum, cudaStream_t s)
{
    hl_update_args a;
    memset(&a, 0, sizeof(a));
    a.w = n->w;
    a.g = n->g;
    a.m = n->m;
    a.v = n->v;
    a.gpart = n->gpart;
    a.gstride = g_stride();
    a.gsum = gsum ? 1 : 0;
    a.n = n_params();
    a.lr = lr;
    a.clip = 1.0f;
    a.nlayers = NET_LAYERS;
    for (int l = 0; l < NET_LAYERS; l++) {
        a.layer[l].off = w_off(l);
        a.layer[l].cout = L_COUT[l];
        a.layer[l].cin = L_CIN[l];
        a.layer[l].flip = L_STRIDE[l] == 1;
        a.layer[l].wf = n->wf[l];
        a.layer[l].wb = l >= 1 ? n->wb[l] : nullptr;
    }
    CKN(hl_launch_update(&a, std::max(n->step, 1), s));
    return HL_NO_ERROR;
}

/* deterministic He-style initialisation (splitmix64 -> Box-Muller) */
static uint64_t sm64(uint64_t *s)
{
    uint64_t z = (*s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

extern "C" int hl_net_num_params(void) { return n_params(); }

extern "C" int hl_net_create(hl_net **out, unsigned long long seed)
{
    if (!out)
        return HL_NULL_POINTER;
    *out = nullptr;
    hl_net *n = new (std::nothrow) hl_net();
    if (!n)
        return HL_OUT_OF_MEM;
    memset(n, 0, sizeof(*n));
    const int np = n_params();
    int rc = HL_NO_ERROR;
    auto fail = [&](int r) { hl_net_destroy(n); return r; };
    if (cudaMalloc(&n->w, np * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&n->g, (np + 2) * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&n->gpart, sizeof(float) * HL_GRAD_COPIES * g_stride()) != cudaSuccess ||
        cudaMalloc(&n->m, np * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&n->v, np * sizeof(float)) != cudaSuccess)
        return fail(HL_OUT_OF_MEM);
    n->loss = n->g + np;
    n->status = reinterpret_cast<int *>(n->loss + 1);
    for (int l = 0; l < NET_LAYERS; l++) {
        const size_t k = (size_t)L_COUT[l] * 9 * L_CIN[l];
        if (cudaMalloc(&n->wf[l], k * sizeof(__nv_bfloat16)) != cudaSuccess ||
            cudaMalloc(&n->wb[l], k * sizeof(__nv_bfloat16)) != cudaSuccess)
            return fail(HL_OUT_OF_MEM);
    }
    std::vector<float> h((size_t)np, 0.0f);
    uint64_t st = seed ^ 0x6A09E667F3BCC909ull;
    for (int l = 0; l < NET_LAYERS; l++) {
        const int fan = 9 * L_CIN[l];
        const float sd = sqrtf(2.0f / (float)fan);
        for (int i = 0; i < L_COUT[l] * fan; i++) {
            double u1 = ((double)(sm64(&st) >> 11) + 0.5) / 9007199254740992.0;
            double u2 = ((double)(sm64(&st) >> 11) + 0.5) / 9007199254740992.0;
            h[(size_t)w_off(l) + i] =
                (float)(sd * sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2));
        }
    }
    h[(size_t)ab_off()] = 1.0f;    /* alpha */
    h[(size_t)ab_off() + 1] = -4.0f;   /* beta: lines are rare */
    if (cudaMemcpy(n->w, h.data(), np * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(n->m, 0, np * sizeof(float)) != cudaSuccess ||
        cudaMemset(n->v, 0, np * sizeof(float)) != cudaSuccess ||
        cudaMemset(n->g, 0, (np + 2) * sizeof(float)) != cudaSuccess)
        return fail(HL_CUDA_ERROR);
    if ((rc = net_update(n, 0.0f, false, 0)) != HL_NO_ERROR || cudaStreamSynchronize(0) != cudaSuccess)
        return fail(rc != HL_NO_ERROR ? rc : HL_CUDA_ERROR);
    *out = n;
    return HL_NO_ERROR;
}

extern "C" int hl_net_destroy(hl_net *n)
{
    if (!n)
        return HL_NULL_POINTER;
    net_free_bufs(n);
    void *p[] = {n->w, n->g, n->gpart, n->m, n->v};
    for (void *q : p)
        if (q)
            cudaFree(q);
    for (int l = 0; l < NET_LAYERS; l++) {
        if (n->wf[l])
            cudaFree(n->wf[l]);
        if (n->wb[l])
            cudaFree(n->wb[l]);
    }
    delete n;
    return HL_NO_ERROR;
}

extern "C" int hl_net_get_params(hl_net *n, float *host)
{
    if (!n || !host)
        return HL_NULL_POINTER;
    CKN(cudaMemcpy(host, n->w, n_params() * sizeof(float), cudaMemcpyDeviceToHost));
    return HL_NO_ERROR;
}

extern "C" int hl_net_get_grads(hl_net *n, float *host)
{
    if (!n || !host)
        return HL_NULL_POINTER;
    CKN(cudaMemcpy(host, n->g, n_params() * sizeof(float), cudaMemcpyDeviceToHost));
    return HL_NO_ERROR;
}

extern "C" int hl_net_set_params(hl_net *n, const float *host)
{
    if (!n || !host)
        return HL_NULL_POINTER;
    CKN(cudaMemcpy(n->w, host, n_params() * sizeof(float), cudaMemcpyHostToDevice));
    CKN(cudaMemset(n->m, 0, n_params() * sizeof(float)));
    CKN(cudaMemset(n->v, 0, n_params() * sizeof(float)));
    n->step = 0;
    int rc = net_update(n, 0.0f, false, 0);
    if (rc != HL_NO_ERROR)
        return rc;
    CKN(cudaStreamSynchronize(0));
    return HL_NO_ERROR;
}

static int conv_layer(hl_net *n, int l, const __nv_bfloat16 *x, int B,
                      __nv_bfloat16 *y, float *y_f32, cudaStream_t s)
{
    hl_conv_args a;
    memset(&a, 0, sizeof(a));
    a.x = x;
    a.w = n->wf[l];
    a.bias = n->w + b_off(l);
    a.y = y;
    a.y_f32 = y_f32;
    a.B = B;
    a.H = a.W = l_in_side(l);
    a.Ho = a.Wo = l_out_side(l);
    a.cin = L_CIN[l];
    a.cout = L_COUT[l];
    a.kreal = 9 * L_CIN[l];
    a.stride = L_STRIDE[l];
    a.relu = L_RELU[l];
    a.w_ready = l > 0;   /* the launch before is the previous layer's */
    a.status = n->status;
    CKN(hl_launch_conv3x3(&a, 0, s));
    return HL_NO_ERROR;
}

/* logits into `logits` (device); the head's sums into n->hsum when training */
static int net_forward(hl_net *n, const __nv_bfloat16 *occ, int B, float *logits, bool train,
                       cudaStream_t s)
{
    int rc;
    const __nv_bfloat16 *x = occ;
    for (int l = 0; l < NET_LAYERS; l++) {
        if (l < NET_LAYERS - 1)
            rc = conv_layer(n, l, x, B, n->act[l], nullptr, s);
        else
            rc = conv_layer(n, l, x, B, nullptr, n->ev, s);
        if (rc != HL_NO_ERROR)
            return rc;
        x = n->act[l];
    }
    CKN(hl_launch_head_fwd(n->ev, n->geo, B, n->w + ab_off(), train ? n->hsum : nullptr,
                           logits, s));
    return HL_NO_ERROR;
}

static int upload_geo(hl_net *n, const hl_coarse_geom *geo, int B, cudaStream_t s)
{
    static_assert(sizeof(hl_coarse_geom) == sizeof(hl_head_geom), "geometry layout");
    CKN(cudaMemcpyAsync(n->geo, geo, (size_t)B * sizeof(hl_head_geom),
                        cudaMemcpyHostToDevice, s));
    return HL_NO_ERROR;
}

extern "C" int hl_net_forward(hl_net *n, const void *occ_dev,
                              const hl_coarse_geom *geo_host, int B,
                              float *logits_dev, void *stream)
{
    if (!n || !occ_dev || !geo_host || !logits_dev)
        return HL_NULL_POINTER;
    if (B <= 0)
        return HL_INVALID_DATA;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    int rc = net_reserve(n, B);
    if (rc != HL_NO_ERROR || (rc = upload_geo(n, geo_host, B, s)) != HL_NO_ERROR)
        return rc;
    return net_forward(n, static_cast<const __nv_bfloat16 *>(occ_dev), B, logits_dev, false, s);
}

/* dW of layer l from the masked gradient of its output: dy (bf16), or the
 * one-channel FP32 gradient dy_f32 of the last layer */
static int layer_dw(hl_net *n, int l, const __nv_bfloat16 *x, const __nv_bfloat16 *dy,
                    const float *dy_f32, int B, cudaStream_t s)
{
    hl_dw_args a;
    memset(&a, 0, sizeof(a));
    a.x = x;
    a.dy = dy;
    a.dy_f32 = dy_f32;
    a.dw = n->gpart + w_off(l);
    a.dw_stride = g_stride();
    a.B = B;
    a.H = a.W = l_in_side(l);
    a.Ho = a.Wo = l_out_side(l);
    a.cin = L_CIN[l];
    a.stride = L_STRIDE[l];
    a.status = n->status;
    CKN(hl_launch_conv_dw(&a, s));
    return HL_NO_ERROR;
}

/* input gradient of layer l (l >= 1) from the bf16 gradient g of its output,
 * masked by the ReLU of layer l - 1, whose bias gradient is its sum */
static int layer_dx(hl_net *n, int l, const __nv_bfloat16 *g, int B,
                    __nv_bfloat16 *dx, cudaStream_t s)
{
    hl_conv_args a;
    memset(&a, 0, sizeof(a));
    a.x = g;
    a.w = n->wb[l];
    a.y = dx;
    a.B = B;
    a.H = a.W = l_out_side(l);
    a.Ho = a.Wo = l_in_side(l);
    a.cin = L_COUT[l];
    a.cout = L_CIN[l];
    a.kreal = 9 * L_COUT[l];
    a.stride = L_STRIDE[l];
    a.w_ready = 1;   /* the weights are the forward pass's */
    a.status = n->status;
    a.mask = n->act[l - 1];
    a.db = n->gpart + b_off(l - 1);
    a.db_stride = g_stride();
    /* stride 1: a convolution with the flipped transposed weights */
    CKN(hl_launch_conv3x3(&a, L_STRIDE[l] == 1 ? 0 : 1, s));
    return HL_NO_ERROR;
}

extern "C" int hl_net_train_step(hl_net *n, const void *occ_dev,
                                 const hl_coarse_geom *geo_host,
                                 const float *target_dev, int B, float lr,
                                 float pos_weight, float *loss_host,
                                 void *stream)
{
    if (!n || !occ_dev || !geo_host || !target_dev)
        return HL_NULL_POINTER;
    if (B <= 0)
        return HL_INVALID_DATA;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const __nv_bfloat16 *occ = static_cast<const __nv_bfloat16 *>(occ_dev);
    int rc = net_reserve(n, B);
    if (rc != HL_NO_ERROR || (rc = upload_geo(n, geo_host, B, s)) != HL_NO_ERROR)
        return rc;
    if ((rc = net_forward(n, occ, B, n->logits, true, s)) != HL_NO_ERROR)
        return rc;
    const int np = n_params();
    CKN(cudaMemsetAsync(n->gpart, 0, sizeof(float) * HL_GRAD_COPIES * g_stride(), s));
    const long long cells = (long long)B * HL_HEAD_T * HL_HEAD_R;
    CKN(hl_launch_bce(n->logits, target_dev, n->hsum, cells, pos_weight, n->dz,
                      n->gpart + ab_off(), n->gpart + np, g_stride(), s));
    CKN(hl_launch_head_bwd(n->dz, NET_EV, n->geo, B, n->w + ab_off(), n->de, n->de_b,
                           n->gpart + b_off(5), g_stride(), s));
    /* layer 5 (32 -> 1, no ReLU): dW from the FP32 gradient, dx from its bf16
     * copy; then layers 4 .. 1, and dW of layer 0 from the input map */
    __nv_bfloat16 *gin = n->gx, *gout = n->gx2;
    if ((rc = layer_dw(n, 5, n->act[4], nullptr, n->de, B, s)) != HL_NO_ERROR ||
        (rc = layer_dx(n, 5, n->de_b, B, gin, s)) != HL_NO_ERROR)
        return rc;
    for (int l = 4; l >= 1; l--) {
        if ((rc = layer_dw(n, l, n->act[l - 1], gin, nullptr, B, s)) != HL_NO_ERROR ||
            (rc = layer_dx(n, l, gin, B, gout, s)) != HL_NO_ERROR)
            return rc;
        std::swap(gin, gout);
    }
    if ((rc = layer_dw(n, 0, occ, gin, nullptr, B, s)) != HL_NO_ERROR)
        return rc;
    n->step++;
    if ((rc = net_update(n, lr, true, s)) != HL_NO_ERROR)
        return rc;
    if (loss_host) {
        int ret[2] = {0, 0};   /* loss (bits), status */
        CKN(cudaMemcpyAsync(ret, n->loss, sizeof(ret), cudaMemcpyDeviceToHost, s));
        CKN(cudaStreamSynchronize(s));
        if (ret[1] != 0)
            return HL_CUDA_ERROR;
        memcpy(loss_host, &ret[0], sizeof(float));
    }
    return HL_NO_ERROR;
}

/* Occupancy maps and coarse geometries of device images: each ROI is pooled
 * in f x f cells, f = max(1, ceil(max(w, h) / 256)), into a 256 x 256 bf16
 * map (cells past the ROI are 0); the evidence cell of the network is 4 f
 * pixels and the coarse rho bins split the image's own rho range. */
extern "C" int hl_occupancy(hl_handle *h, const hl_image_desc *imgs, int nimg,
                            void *occ_dev, hl_coarse_geom *geo_host,
                            void *stream)
{
    if (!h || !imgs || !occ_dev || !geo_host)
        return HL_NULL_POINTER;
    if (nimg <= 0)
        return HL_INVALID_DATA;
    std::vector<hl_pool_img> pi((size_t)nimg);
    for (int i = 0; i < nimg; i++) {
        const hl_image_desc &d = imgs[i];
        if (!d.data)
            return HL_NULL_POINTER;
        if (d.roi_x1 < 0 || d.roi_y1 < 0 || d.roi_x2 > d.width || d.roi_y2 > d.height ||
            d.roi_x2 <= d.roi_x1 || d.roi_y2 <= d.roi_y1)
            return HL_INVALID_DATA;
        const int w = d.roi_x2 - d.roi_x1, hh = d.roi_y2 - d.roi_y1;
        const int f = std::max(1, (std::max(w, hh) + NET_IN - 1) / NET_IN);
        pi[i].base = d.data + (size_t)d.roi_y1 * d.pitch + d.roi_x1;
        pi[i].pitch = (long)d.pitch;
        pi[i].w = w;
        pi[i].h = hh;
        pi[i].factor = f;
        pi[i].pad = 0;
        hl_geom g;
        int rc = hl_geometry(h, w, hh, &g);
        if (rc != HL_NO_ERROR)
            return rc;
        hl_coarse_geom &cg = geo_host[i];
        cg.cell = (float)(4 * f);
        cg.rho_min = (float)g.rho_min;
        cg.inv_rw = (float)HL_HEAD_R / (float)g.numrho;
        const int ph = (hh + f - 1) / f, pw = (w + f - 1) / f;
        cg.qh = (ph + 3) / 4;
        cg.qw = (pw + 3) / 4;
        cg.pad = 0;
    }
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    hl_pool_img *d_pi = nullptr;
    CKN(cudaMallocAsync(&d_pi, sizeof(hl_pool_img) * nimg, s));
    cudaError_t e = cudaMemcpyAsync(d_pi, pi.data(), sizeof(hl_pool_img) * nimg,
                                    cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
        e = hl_launch_pool(d_pi, nimg, NET_IN, static_cast<__nv_bfloat16 *>(occ_dev), s);
    cudaFreeAsync(d_pi, s);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(s);
    return cnn_err(e);
}

/* Forward pass for the proposal pipeline: geometry already on the device. */
int hl_net_run(hl_net *n, const __nv_bfloat16 *occ, const hl_head_geom *geo_dev,
               int B, const float **logits, cudaStream_t s)
{
    int rc = net_reserve(n, B);
    if (rc != HL_NO_ERROR)
        return rc;
    CKN(cudaMemcpyAsync(n->geo, geo_dev, (size_t)B * sizeof(hl_head_geom),
                        cudaMemcpyDeviceToDevice, s));
    if ((rc = net_forward(n, occ, B, n->logits, false, s)) != HL_NO_ERROR)
        return rc;
    *logits = n->logits;
    return HL_NO_ERROR;
}

int hl_net_status(hl_net *n, int *st, cudaStream_t s)
{
    CKN(cudaMemcpyAsync(st, n->status, sizeof(int), cudaMemcpyDeviceToHost, s));
    return HL_NO_ERROR;
}
