/*
 * hl_cnn.cu -- the proposal network's kernels: 3x3 convolutions as implicit
 * GEMMs on the 5th-generation tensor cores (tcgen05.mma, BF16 operands in
 * shared memory, FP32 accumulators in tensor memory), their backward passes,
 * the occupancy pooling and the fixed coarse Hough head.
 *
 * The reference has no learned component; this is the proposal stage of the
 * plain method's accelerated variant: a small CNN reads an average-pooled
 * edge map and predicts which coarse (theta, rho) cells hold lines, and the
 * exact int32 vote then runs only in those cells (hl_proposal.cpp).
 *
 * Activations are NHWC bfloat16 with C = 32 (64 bytes per pixel), the input
 * map is NHWC with C = 1.  Weights are [Cout][K] bfloat16 with K = tap * Cin
 * + ci (tap = ky * 3 + kx), K-major, so that one GEMM row of the weight
 * operand is one output channel.
 *
 * Implicit GEMM, CTAs of 128 threads, one M = 128 tile of 8 x 16 output
 * pixels at a time: D[128 x N] = sum over the taps of A_tap[128 x 32] *
 * B_tap[N x 32]^T.  The input tile and its halo are copied into shared memory
 * once (cp.async, zero outside the image) as rows of four channel planes,
 * [row][8-channel group][pixel][8 channels]: 8 neighbouring pixels of a plane
 * are 128 contiguous bytes, one core matrix of the no-swizzle K-major layout,
 * whichever pixel they start at.  So every tap's A operand is the same halo
 * at another start address (LBO one plane, SBO one output row), and nothing
 * is gathered per tap.  One thread issues the tcgen05.mma in tap order (M = 128,
 * N = 32 or 16, K = 16) into TMEM and commits them to an mbarrier; the next
 * tile's copies are issued behind them; each warp reads its 32 TMEM lanes
 * (tcgen05.ld 32x32b), runs the epilogue and stores whole 512-byte rows.
 */
#include "hl_internal.h"
#include "hl_cnn.h"
#include "hl_device.cuh"

#include <cuda_bf16.h>

#define FULL 0xffffffffu
#define CNN_THREADS 128
#define CNN_TILE_M 128
#define CNN_WAIT_LIMIT (1 << 22)

/* ---- tcgen05 / mbarrier primitives ------------------------------------- */
__device__ __forceinline__ unsigned cnn_smem_u32(const void *p)
{
    return (unsigned)__cvta_generic_to_shared(p);
}

/* Shared-memory matrix descriptor, no swizzle, K-major: start address,
 * leading-dimension byte offset (between the two 8-element K groups of one
 * MMA), stride byte offset (between 8-row groups), descriptor version 1. */
__device__ __forceinline__ unsigned long long smem_desc(unsigned addr,
                                                        unsigned lbo,
                                                        unsigned sbo)
{
    unsigned long long d = 0;
    d |= (unsigned long long)((addr >> 4) & 0x3fffu);
    d |= (unsigned long long)((lbo >> 4) & 0x3fffu) << 16;
    d |= (unsigned long long)((sbo >> 4) & 0x3fffu) << 32;
    d |= 1ull << 46;   /* version */
    /* base offset 0, lbo mode 0, layout type 0 = no swizzle */
    return d;
}

/* Instruction descriptor of kind::f16: D f32, A and B bf16, both K-major,
 * no negation, N and M as given. */
__host__ __device__ constexpr unsigned mma_idesc(int M, int N)
{
    return (1u << 4)                       /* D format f32 */
           | (1u << 7)                     /* A format bf16 */
           | (1u << 10)                    /* B format bf16 */
           | ((unsigned)(N >> 3) << 17)    /* N / 8 */
           | ((unsigned)(M >> 4) << 24);   /* M / 16 */
}

__device__ __forceinline__ void cnn_mbar_init(unsigned long long *bar, unsigned n)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(cnn_smem_u32(bar)),
                 "r"(n)
                 : "memory");
}

__device__ __forceinline__ bool cnn_mbar_wait(unsigned long long *bar,
                                              unsigned parity)
{
    const unsigned a = cnn_smem_u32(bar);
    for (int i = 0; i < CNN_WAIT_LIMIT; i++) {
        unsigned ok;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], "
            "%2; selp.u32 %0, 1, 0, p; }"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok)
            return true;
    }
    return false;
}

__device__ __forceinline__ void tmem_alloc(unsigned *dst_smem, int cols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(cnn_smem_u32(dst_smem)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(unsigned taddr, int cols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols)
                 : "memory");
}

__device__ __forceinline__ void umma_f16(unsigned tmem_d, unsigned long long adesc,
                                         unsigned long long bdesc, unsigned idesc,
                                         int accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

/* one lane of a converged warp: the branch stays warp-uniform, so descriptors
 * are built in uniform registers */
__device__ __forceinline__ bool elect_one()
{
    unsigned p;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void umma_commit(unsigned long long *bar)
{
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
        ::"r"(cnn_smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

/* 32 consecutive fp32 columns of this thread's TMEM lane */
__device__ __forceinline__ void tmem_ld32(unsigned taddr, float (&v)[32])
{
    unsigned r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
          "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]),
          "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
          "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++)
        v[i] = __uint_as_float(r[i]);
}

/* ---- the convolution ----------------------------------------------------- */

/* output tile: 8 x 16 pixels, GEMM row m = pixel (m / 8, m % 8) */
#define CONV_TX 8
#define CONV_TY 16

/* Kinds of the 32-channel convolution. */
enum { CONV_S1 = 0,     /* stride 1 */
       CONV_S2 = 1,     /* stride 2 */
       CONV_T2 = 2 };   /* x-gradient of a stride-2 convolution:
                           dx[p] = sum w * dy[(p + 1 - tap) / 2] */

/* The halo of a tile in shared memory: ROWS x COLS input pixels, a plane row
 * of P bytes per (row, 8-channel group).  CONV_S2 keeps even and odd columns
 * in two halves (HALF bytes apart), so that the 8 pixels of an output row,
 * two columns apart, are neighbours.  A half starts 64 bytes off the banks of
 * the other and P is 32 or 16 bytes off a multiple of 128, so the copies of
 * 8 lanes (2 pixels x 4 planes) hit all banks. */
template <int MODE> struct ConvHalo;
template <> struct ConvHalo<CONV_S1> {
    static constexpr int COLS = 10, ROWS = 18, P = 160, HALF = 0, BYTES = 18 * 4 * 160, NST = 2;
    static constexpr int TMEM_COLS = 32, CTAS = 4;
};
template <> struct ConvHalo<CONV_S2> {
    static constexpr int COLS = 17, ROWS = 33, P = 144, HALF = 33 * 4 * 144,
                         BYTES = 2 * 33 * 4 * 144, NST = 1;
    static constexpr int TMEM_COLS = 32, CTAS = 3;
};
template <> struct ConvHalo<CONV_T2> {
    static constexpr int COLS = 9, ROWS = 17, P = 144, HALF = 0, BYTES = 17 * 4 * 144, NST = 2;
    static constexpr int TMEM_COLS = 128, CTAS = 4;
};

/* B operand: core matrix (row group g, K group q) at (g * KG + q) * 128 bytes,
 * so LBO = 128 and SBO = KG * 128. */
template <int KG, int NROWS, int ABYTES>
struct ConvSmem {
    alignas(128) unsigned char b[NROWS / 8][KG][128];
    alignas(128) unsigned char a[ABYTES];
    alignas(128) unsigned char out[CNN_THREADS / 32][32 * 64];   /* a warp's output pixels */
    alignas(16) float bias[32];
    unsigned long long bar;
    unsigned tmem;
};

/* weights -> B operand: row n = output channel, K group q = 8 consecutive k;
 * rows n >= cout and k >= kreal are zero */
template <int KG, int N>
__device__ __forceinline__ void conv_weights(unsigned char (*b)[KG][128], const hl_conv_args &a)
{
    const bool vec = a.kreal % 8 == 0 && (((uintptr_t)a.w) & 15u) == 0;
    constexpr int NE = N * KG / CNN_THREADS + (N * KG % CNN_THREADS != 0);
    uint4 v[NE];   /* every load in flight before the first store */
#pragma unroll
    for (int i = 0; i < NE; i++) {
        /* 8 lanes take 4 channels x 2 K groups: whole sectors read, stores at
         * most two to a bank */
        const int e = threadIdx.x + i * CNN_THREADS;
        const int q = ((e >> 3) % (KG / 2)) * 2 + (e & 1);
        const int n = ((e >> 1) & 3) + 4 * (e / (4 * KG));
        v[i] = make_uint4(0u, 0u, 0u, 0u);
        if (e < N * KG && vec) {
            if (n < a.cout && q * 8 < a.kreal)
                v[i] = *reinterpret_cast<const uint4 *>(a.w + (size_t)n * a.kreal + q * 8);
        } else if (e < N * KG) {
            __nv_bfloat16 v8[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int k = q * 8 + j;
                const bool ok = n < a.cout && k < a.kreal;
                v8[j] = ok ? a.w[(size_t)n * a.kreal + k] : __float2bfloat16(0.0f);
            }
            v[i] = *reinterpret_cast<const uint4 *>(v8);
        }
    }
#pragma unroll
    for (int i = 0; i < NE; i++) {
        const int e = threadIdx.x + i * CNN_THREADS;
        const int q = ((e >> 3) % (KG / 2)) * 2 + (e & 1);
        const int n = ((e >> 1) & 3) + 4 * (e / (4 * KG));
        if (e < N * KG)
            *reinterpret_cast<uint4 *>(&b[n >> 3][q][(n & 7) * 16]) = v[i];
    }
}

/* A tile of the output (CONV_T2: of the input): its image and first pixel. */
struct ConvTile {
    int b, y0, x0;
};
/* The tiles blockIdx.x, blockIdx.x + gridDim.x, ...: divisions once, then the
 * grid's own (x, y, image) step with carries. */
template <int TX, int TY>
struct ConvTiles {
    int tx_n, ty_n, x, y, b, dx, dy, db;
    __device__ __forceinline__ ConvTiles(int tx, int ty) : tx_n(tx), ty_n(ty)
    {
        const int r = blockIdx.x / tx, gr = gridDim.x / tx;
        x = blockIdx.x - r * tx;
        b = r / ty;
        y = r - b * ty;
        dx = gridDim.x - gr * tx;
        db = gr / ty;
        dy = gr - db * ty;
    }
    __device__ __forceinline__ ConvTile get() const
    {
        ConvTile t;
        t.b = b;
        t.y0 = y * TY;
        t.x0 = x * TX;
        return t;
    }
    __device__ __forceinline__ void next()
    {
        x += dx;
        y += dy;
        b += db;
        if (x >= tx_n) {
            x -= tx_n;
            y++;
        }
        if (y >= ty_n) {
            y -= ty_n;
            b++;
        }
    }
};

/* Start of a convolution kernel: TMEM columns and the mbarrier.  It comes
 * before hl_pdl_begin lets the next launch in, so a waiting successor never
 * holds columns this kernel still needs. */
__device__ __forceinline__ unsigned conv_begin(unsigned *tmem_s, unsigned long long *bar,
                                               int cols)
{
    if (threadIdx.x < 32)
        tmem_alloc(tmem_s, cols);
    if (threadIdx.x == 0) {
        cnn_mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    return *tmem_s;
}

/* two floats -> packed bf16 (the first in the low half) */
__device__ __forceinline__ unsigned pack_bf16(float lo, float hi)
{
    const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned *>(&p);
}

/* v with the halves zeroed where m's bf16 half is not above zero (the ReLU
 * mask), the kept values added to s0 (low half) and s1 */
__device__ __forceinline__ unsigned mask_bf16(unsigned v, unsigned m, float &s0, float &s1)
{
    if (!(__uint_as_float(m << 16) > 0.0f))
        v &= 0xffff0000u;
    if (!(__uint_as_float(m & 0xffff0000u) > 0.0f))
        v &= 0x0000ffffu;
    s0 += __uint_as_float(v << 16);
    s1 += __uint_as_float(v & 0xffff0000u);
    return v;
}

/* Epilogue of a warp's 32 pixels (its TMEM lanes; columns tcol ..): bias and
 * ReLU in fp32, bf16 rounding, then through the warp's staging buffer so that
 * 8 neighbouring output pixels leave as one 512-byte store.  Tile row r (8
 * pixels) goes to output row oy0 + r * osy, columns ox0 + x * osx.  GRAD: the
 * values are an input gradient; they are masked by the layer's ReLU output
 * a.mask on the way out and summed over the pixels (its bias gradient), lane
 * l holding channels 8 (l % 4) .. in db. */
template <bool GRAD>
__device__ __forceinline__ void conv_epilogue(const hl_conv_args &a, unsigned tcol,
                                              unsigned char *stage, const float *bias, int bimg,
                                              int oy0, int ox0, int osy, int osx, float (&db)[8])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float v[32];
    tmem_ld32(tcol + ((unsigned)(32 * warp) << 16), v);
    if (a.y_f32) {
        const int m = 32 * warp + lane;
        const int oy = oy0 + (m >> 3) * osy, ox = ox0 + (m & 7) * osx;
        if (oy < a.Ho && ox < a.Wo) {
            float o = v[0] + bias[0];
            if (a.relu)
                o = fmaxf(o, 0.0f);
            a.y_f32[((size_t)bimg * a.Ho + oy) * a.Wo + ox] = o;
        }
        return;
    }
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const float4 bb = reinterpret_cast<const float4 *>(bias)[c];
        v[4 * c] += bb.x;
        v[4 * c + 1] += bb.y;
        v[4 * c + 2] += bb.z;
        v[4 * c + 3] += bb.w;
    }
    if (a.relu) {
#pragma unroll
        for (int c = 0; c < 32; c++)
            v[c] = fmaxf(v[c], 0.0f);
    }
    if (a.cout < 32) {
#pragma unroll
        for (int c = 0; c < 32; c++)
            v[c] = c < a.cout ? v[c] : 0.0f;
    }
#pragma unroll
    for (int c = 0; c < 4; c++)
        /* chunk c of pixel p at 16-byte slot 4 p + (c ^ (p / 2) % 4) */
        *reinterpret_cast<uint4 *>(stage + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) =
            make_uint4(pack_bf16(v[8 * c], v[8 * c + 1]), pack_bf16(v[8 * c + 2], v[8 * c + 3]),
                       pack_bf16(v[8 * c + 4], v[8 * c + 5]),
                       pack_bf16(v[8 * c + 6], v[8 * c + 7]));
    __syncwarp();
    const int x = lane >> 2, q = lane & 3;
    const int ox = ox0 + x * osx;
#pragma unroll
    for (int it = 0; it < 4; it++) {
        const int p = it * 8 + x;
        uint4 o = *reinterpret_cast<const uint4 *>(stage + p * 64 + ((q ^ ((p >> 1) & 3)) << 4));
        const int oy = oy0 + (4 * warp + it) * osy;
        if (oy < a.Ho && ox < a.Wo) {
            const size_t at = (((size_t)bimg * a.Ho + oy) * a.Wo + ox) * 32 + q * 8;
            if (GRAD) {
                const uint4 m = *reinterpret_cast<const uint4 *>(a.mask + at);
                o.x = mask_bf16(o.x, m.x, db[0], db[1]);
                o.y = mask_bf16(o.y, m.y, db[2], db[3]);
                o.z = mask_bf16(o.z, m.z, db[4], db[5]);
                o.w = mask_bf16(o.w, m.w, db[6], db[7]);
            }
            *reinterpret_cast<uint4 *>(a.y + at) = o;
        }
    }
    __syncwarp();
}

/* the CTA's bias-gradient sums (conv_epilogue's db) added to its copy of a.db:
 * lanes, then warps (s: 4 x 32 floats), then one 32-channel reduction */
__device__ __forceinline__ void conv_add_db(const hl_conv_args &a, float (&db)[8], float *s)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
        for (int o = 4; o < 32; o <<= 1)
            db[j] += __shfl_xor_sync(FULL, db[j], o);
    __syncthreads();
    if (lane < 4)
#pragma unroll
        for (int j = 0; j < 8; j++)
            s[warp * 32 + lane * 8 + j] = db[j];
    __syncthreads();
    if (warp == 0 && lane < a.cout)
        atomicAdd(a.db + (size_t)(blockIdx.x % HL_GRAD_COPIES) * a.db_stride + lane,
                  (s[lane] + s[32 + lane]) + (s[64 + lane] + s[96 + lane]));
}

/* 32 input channels.  What bounds it: shared memory -- the tensor cores read
 * each pixel once a tap (18 MMAs x 5 KB of operands, about 720 cycles a tile,
 * and 460 of copies and staging); the MMAs themselves are busy 12%.  Several
 * CTAs an SM overlap one tile's copies and epilogue with another's MMAs, and
 * weights that are ready are read while the launch before still runs.  64
 * images of 64 x 64, stride 1, ncu: 15.5 us a launch, against 55.0 us when
 * every tap was gathered into an im2col tile; stride 2 (bound by the 67 MB it
 * reads) 28.9 against 55.5, one-channel output 12.9 against 41.5. */
template <int N, int MODE, bool GRAD>
__global__ void __launch_bounds__(CNN_THREADS)
hl_conv32_kernel(hl_conv_args a)
{
    float db[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    using H = ConvHalo<MODE>;
    constexpr int KG = 36;
    extern __shared__ __align__(128) unsigned char conv_raw[];
    typedef ConvSmem<KG, N, H::NST * ((H::BYTES + 127) / 128 * 128)> Smem;
    Smem &sm = *reinterpret_cast<Smem *>(conv_raw);
    constexpr unsigned STAGE = (H::BYTES + 127) / 128 * 128;
    const int tid = threadIdx.x;
    const unsigned tmem = conv_begin(&sm.tmem, &sm.bar, H::TMEM_COLS);

    /* weights written before the previous launch began are read while it
     * still runs */
    if (!a.w_ready)
        hl_pdl_begin();
    conv_weights<KG, N>(sm.b, a);
    if (tid < 32)
        sm.bias[tid] = (a.bias && tid < a.cout) ? a.bias[tid] : 0.0f;
    if (a.w_ready)
        hl_pdl_begin();
    /* tiles cover the output (CONV_T2: the input, four outputs a position) */
    const int EX = MODE == CONV_T2 ? a.W : a.Wo, EY = MODE == CONV_T2 ? a.H : a.Ho;
    const int tx_n = (EX + CONV_TX - 1) / CONV_TX, ty_n = (EY + CONV_TY - 1) / CONV_TY;
    const int ntiles = a.B * tx_n * ty_n;
    const unsigned abase = cnn_smem_u32(sm.a), bbase = cnn_smem_u32(sm.b);

    /* a thread copies plane q of every 32nd halo pixel */
    auto load = [&](const ConvTile &t, unsigned st) {
        constexpr int S = MODE == CONV_S2 ? 2 : 1;
        const int iy0 = t.y0 * S - (MODE == CONV_T2 ? 0 : 1);
        const int ix0 = t.x0 * S - (MODE == CONV_T2 ? 0 : 1);
        const int q = tid & 3;
        const __nv_bfloat16 *x = a.x + (size_t)t.b * a.H * a.W * 32 + q * 8;
        int hy = (tid >> 2) / H::COLS, hx = (tid >> 2) % H::COLS;
        for (int px = tid >> 2; px < H::ROWS * H::COLS; px += CNN_THREADS / 4) {
            const int iy = iy0 + hy, ix = ix0 + hx;
            const bool ok = (unsigned)iy < (unsigned)a.H && (unsigned)ix < (unsigned)a.W;
            const __nv_bfloat16 *src = ok ? x + (size_t)(iy * a.W + ix) * 32 : a.x;
            const unsigned dst =
                abase + st + (unsigned)((hy * 4 + q) * H::P) +
                (MODE == CONV_S2 ? (unsigned)((hx & 1) * H::HALF + (hx >> 1) * 16)
                                 : (unsigned)(hx * 16));
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                         ::"r"(dst), "l"(src), "r"(ok ? 16 : 0)
                         : "memory");
            hx += 32 % H::COLS;
            hy += 32 / H::COLS;
            if (hx >= H::COLS) {
                hx -= H::COLS;
                hy++;
            }
        }
    };

    unsigned phase = 0, st = 0;
    bool failed = false;
    ConvTiles<CONV_TX, CONV_TY> walk(tx_n, ty_n);
    ConvTile cur = walk.get();
    if ((int)blockIdx.x < ntiles)
        load(cur, 0);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        /* the copies (and the weights) visible to the tensor cores */
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (__syncthreads_or(failed))
            break;
        if (tid < 32 && elect_one()) {
            tmem_fence_after();
            constexpr unsigned idesc = mma_idesc(CNN_TILE_M, N);
            constexpr unsigned sbo = (MODE == CONV_S2 ? 8 : 4) * H::P;
            /* descriptors of tap 0; a tap's differ by a constant in the
             * 16-byte address field */
            const unsigned long long ad0 = smem_desc(abase + st, H::P, sbo);
            const unsigned long long bd0 = smem_desc(bbase, 128, KG * 128);
            /* CONV_T2: output parity class cls = 2 py + px; others one class */
#pragma unroll
            for (int cls = 0; cls < (MODE == CONV_T2 ? 4 : 1); cls++) {
                bool first = true;
#pragma unroll
                for (int tap = 0; tap < 9; tap++) {
                    const int ky = tap / 3, kx = tap % 3;
                    unsigned off;
                    if (MODE == CONV_T2) {
                        /* rows with (p + 1 - tap) odd take no tap; an even row
                         * takes ky = 1 at j, an odd one ky = 0 at j + 1 and
                         * ky = 2 at j */
                        if (((cls >> 1) + 1 - ky) & 1 || ((cls & 1) + 1 - kx) & 1)
                            continue;
                        const int dy = ((cls >> 1) + 1 - ky) >> 1, dx = ((cls & 1) + 1 - kx) >> 1;
                        off = (unsigned)(dy * 4 * H::P + dx * 16);
                    } else if (MODE == CONV_S2) {
                        off = (unsigned)(ky * 4 * H::P + (kx & 1) * H::HALF + (kx >> 1) * 16);
                    } else {
                        off = (unsigned)(ky * 4 * H::P + kx * 16);
                    }
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        umma_f16(tmem + (unsigned)(cls * 32),
                                 ad0 + ((off + (unsigned)(2 * h * H::P)) >> 4),
                                 bd0 + (unsigned)((tap * 2 + h) * 16), idesc, !first);
                        first = false;
                    }
                }
            }
            umma_commit(&sm.bar);
        }
        __syncwarp();
        const int next = tile + (int)gridDim.x;
        walk.next();
        const ConvTile nt = walk.get();
        if (H::NST == 2 && next < ntiles)
            load(nt, st ^ STAGE);
        const bool got = cnn_mbar_wait(&sm.bar, phase);
        phase ^= 1u;
        tmem_fence_after();
        if (!got) {
            failed = true;
            if ((tid & 31) == 0)
                atomicOr(a.status, HL_ST_CNN_TIMEOUT);
            continue;
        }
        if (H::NST == 1 && next < ntiles)
            load(nt, 0);   /* the MMAs have read the halo */
        else if (H::NST == 2)
            st ^= STAGE;
        if (MODE == CONV_T2) {
#pragma unroll 1
            for (int cls = 0; cls < 4; cls++)
                conv_epilogue<GRAD>(a, tmem + (unsigned)(cls * 32), sm.out[tid >> 5], sm.bias,
                                    cur.b, 2 * cur.y0 + (cls >> 1), 2 * cur.x0 + (cls & 1), 2, 2,
                                    db);
        } else {
            conv_epilogue<GRAD>(a, tmem, sm.out[tid >> 5], sm.bias, cur.b, cur.y0, cur.x0, 1, 1,
                                db);
        }
        cur = nt;
        /* TMEM reads done before the next tile's MMAs (ordered by the
         * barrier at the loop's top) */
        tmem_fence_before();
    }
    if (failed) {
        /* a commit that never arrived: nothing more is issued; wait once
         * more (bounded) so no MMA still writes the TMEM being released */
        cnn_mbar_wait(&sm.bar, phase ^ 1u);
    }
    if (GRAD)
        conv_add_db(a, db, reinterpret_cast<float *>(sm.out));
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (tid < 32)
        tmem_dealloc(tmem, H::TMEM_COLS);
}

/* One input channel, stride 1 or 2: K = 16 (9 taps, then zeros), a thread
 * gathers the 9 values of its output pixel into its row of A; the next tile's
 * values are loaded behind the MMA.  Bound by its epilogue's instructions and
 * the output's 64 bytes a pixel: 64 maps of 256 x 256, stride 2, 23.8 us
 * (46.6 us before). */
template <bool GRAD>
__global__ void __launch_bounds__(CNN_THREADS)
hl_conv1_kernel(hl_conv_args a)
{
    float db[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    constexpr int KG = 2, N = 32;
    extern __shared__ __align__(128) unsigned char conv_raw[];
    typedef ConvSmem<KG, N, CNN_TILE_M * 32> Smem;
    Smem &sm = *reinterpret_cast<Smem *>(conv_raw);
    const int tid = threadIdx.x;
    const unsigned tmem = conv_begin(&sm.tmem, &sm.bar, 32);
    hl_pdl_begin();
    conv_weights<KG, N>(sm.b, a);
    if (tid < 32)
        sm.bias[tid] = (a.bias && tid < a.cout) ? a.bias[tid] : 0.0f;
    const int tx_n = (a.Wo + CONV_TX - 1) / CONV_TX, ty_n = (a.Ho + CONV_TY - 1) / CONV_TY;
    const int ntiles = a.B * tx_n * ty_n;
    const unsigned abase = cnn_smem_u32(sm.a), bbase = cnn_smem_u32(sm.b);

    unsigned short v[9];   /* the pixel's taps, as bf16 bits */
    auto gather = [&](const ConvTile &t) {
        const int iy0 = (t.y0 + (tid >> 3)) * a.stride - 1;
        const int ix0 = (t.x0 + (tid & 7)) * a.stride - 1;
        const unsigned short *x =
            reinterpret_cast<const unsigned short *>(a.x) + (size_t)t.b * a.H * a.W;
        bool okx[3];
#pragma unroll
        for (int kx = 0; kx < 3; kx++)
            okx[kx] = (unsigned)(ix0 + kx) < (unsigned)a.W;
#pragma unroll
        for (int ky = 0; ky < 3; ky++) {
            const bool oky = (unsigned)(iy0 + ky) < (unsigned)a.H;
            const unsigned short *row = x + (ptrdiff_t)(iy0 + ky) * a.W + ix0;
#pragma unroll
            for (int kx = 0; kx < 3; kx++)
                v[3 * ky + kx] = oky && okx[kx] ? row[kx] : (unsigned short)0;
        }
    };
    unsigned phase = 0;
    bool failed = false;
    ConvTiles<CONV_TX, CONV_TY> walk(tx_n, ty_n);
    ConvTile cur = walk.get();
    if ((int)blockIdx.x < ntiles)
        gather(cur);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        unsigned char *row = sm.a + (tid >> 3) * 256 + (tid & 7) * 16;
        *reinterpret_cast<uint4 *>(row) =
            make_uint4(v[0] | ((unsigned)v[1] << 16), v[2] | ((unsigned)v[3] << 16),
                       v[4] | ((unsigned)v[5] << 16), v[6] | ((unsigned)v[7] << 16));
        *reinterpret_cast<uint4 *>(row + 128) = make_uint4(v[8], 0u, 0u, 0u);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (__syncthreads_or(failed))
            break;
        if (tid < 32 && elect_one()) {
            tmem_fence_after();
            umma_f16(tmem, smem_desc(abase, 128, 256), smem_desc(bbase, 128, 256),
                     mma_idesc(CNN_TILE_M, N), 0);
            umma_commit(&sm.bar);
        }
        __syncwarp();
        const int next = tile + (int)gridDim.x;
        walk.next();
        const ConvTile nt = walk.get();
        if (next < ntiles)
            gather(nt);
        const bool got = cnn_mbar_wait(&sm.bar, phase);
        phase ^= 1u;
        tmem_fence_after();
        if (!got) {
            failed = true;
            if ((tid & 31) == 0)
                atomicOr(a.status, HL_ST_CNN_TIMEOUT);
            continue;
        }
        conv_epilogue<GRAD>(a, tmem, sm.out[tid >> 5], sm.bias, cur.b, cur.y0, cur.x0, 1, 1, db);
        cur = nt;
        tmem_fence_before();
    }
    if (failed)
        cnn_mbar_wait(&sm.bar, phase ^ 1u);   /* as in hl_conv32_kernel */
    if (GRAD)
        conv_add_db(a, db, reinterpret_cast<float *>(sm.out));
    __syncthreads();
    if (tid < 32)
        tmem_dealloc(tmem, 32);
}

template <typename K>
static cudaError_t launch_conv(K kernel, size_t smem, long long ntiles, int ctas_per_sm,
                               const hl_conv_args *a, cudaStream_t s)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess)
        return e;
    if (ntiles > 0x7fffffffLL)
        return cudaErrorInvalidValue;
    const int grid = (int)std::max(1LL, std::min(ntiles, (long long)sms * ctas_per_sm));
    return hl_launch_pdl(kernel, dim3(grid), dim3(CNN_THREADS), smem, s, false, *a);
}

template <int N, int MODE, bool GRAD>
static cudaError_t launch_conv32(const hl_conv_args *a, cudaStream_t s)
{
    typedef ConvHalo<MODE> H;
    typedef ConvSmem<36, N, H::NST * ((H::BYTES + 127) / 128 * 128)> Smem;
    const int ex = MODE == CONV_T2 ? a->W : a->Wo, ey = MODE == CONV_T2 ? a->H : a->Ho;
    const long long nt = (long long)a->B * ((ex + CONV_TX - 1) / CONV_TX) *
                         ((ey + CONV_TY - 1) / CONV_TY);
    return launch_conv(hl_conv32_kernel<N, MODE, GRAD>, sizeof(Smem), nt, H::CTAS, a, s);
}

cudaError_t hl_launch_conv3x3(const hl_conv_args *a, int mode, cudaStream_t s)
{
    const bool grad = a->mask != nullptr;   /* an input gradient of the network */
    if (a->cin == 1 && a->cout <= 32 && mode == 0) {
        const long long nt = (long long)a->B * ((a->Wo + CONV_TX - 1) / CONV_TX) *
                             ((a->Ho + CONV_TY - 1) / CONV_TY);
        const size_t smem = sizeof(ConvSmem<2, 32, CNN_TILE_M * 32>);
        return grad ? launch_conv(hl_conv1_kernel<true>, smem, nt, 8, a, s)
                    : launch_conv(hl_conv1_kernel<false>, smem, nt, 8, a, s);
    }
    if (a->cin != 32 || a->cout > 32)
        return cudaErrorInvalidValue;
    if (mode == 1)
        return grad ? launch_conv32<32, CONV_T2, true>(a, s)
                    : launch_conv32<32, CONV_T2, false>(a, s);
    if (mode != 0)
        return cudaErrorInvalidValue;
    if (a->stride == 2)
        return a->cout <= 16 ? launch_conv32<16, CONV_S2, false>(a, s)
                             : launch_conv32<32, CONV_S2, false>(a, s);
    if (grad)
        return launch_conv32<32, CONV_S1, true>(a, s);
    return a->cout <= 16 ? launch_conv32<16, CONV_S1, false>(a, s)
                         : launch_conv32<32, CONV_S1, false>(a, s);
}

/* ---- occupancy pooling ---------------------------------------------------- */

/* out[b][i][j] (side x side, bf16) = fraction of 255-pixels in the f x f
 * block (i * f.., j * f..) of image b's ROI; blocks past the ROI count as
 * empty.  One thread per output cell.  Cells whose rows are whole words (f a
 * multiple of 4, rows aligned alike; of 8 for the wider one) read them row after
 * row with eight rows' loads in flight, the others four bytes or one at a time.
 * Bound by the images' bytes: 134 MB (32 images of 2048 x 2048) in 25 us (48 us
 * with four bytes a load, one row after the other). */
template <typename V>
__device__ __forceinline__ int pool_words(const uint8_t *p, long pitch, int f, int rows)
{
    int cnt = 0;
    for (int x = 0; x < f; x += (int)sizeof(V)) {
#pragma unroll 8
        for (int y = 0; y < rows; y++) {
            const V v = __ldcs(reinterpret_cast<const V *>(p + (size_t)y * pitch + x));
            const unsigned *w = reinterpret_cast<const unsigned *>(&v);
#pragma unroll
            for (int q = 0; q < (int)(sizeof(V) / 4); q++)
                cnt += __popc(ff_flags(w[q]));
        }
    }
    return cnt;
}

__global__ void __launch_bounds__(256)
hl_pool_kernel(const hl_pool_img *imgs, int nimg, int side, __nv_bfloat16 *out)
{
    const int per = side * side;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
         e < (size_t)nimg * per; e += (size_t)gridDim.x * blockDim.x) {
        const int b = (int)(e / per), r = (int)(e % per);
        const int i = r / side, j = r % side;
        const hl_pool_img im = imgs[b];
        const int f = im.factor;
        int cnt = 0;
        const int y0 = i * f, x0 = j * f;
        const int x1 = min(x0 + f, im.w), y1 = min(y0 + f, im.h);
        const uint8_t *p = im.base + (size_t)y0 * im.pitch + x0;
        const unsigned mis = (unsigned)((uintptr_t)p | (uintptr_t)im.pitch | (unsigned)f);
        if (x0 + f <= im.w && (mis & 7u) == 0) {
            cnt = pool_words<uint2>(p, im.pitch, f, max(y1 - y0, 0));
        } else if (x0 + f <= im.w && (mis & 3u) == 0) {
            cnt = pool_words<unsigned>(p, im.pitch, f, max(y1 - y0, 0));
        } else {
            for (int y = y0; y < y1; y++) {
                const uint8_t *row = im.base + (size_t)y * im.pitch;
                int x = x0;
                if ((((uintptr_t)(row + x)) & 3u) == 0)
                    for (; x + 4 <= x1; x += 4)
                        cnt += __popc(ff_flags(*reinterpret_cast<const unsigned *>(row + x)));
                for (; x < x1; x++)
                    cnt += row[x] == 255;
            }
        }
        out[e] = __float2bfloat16((float)cnt / (float)(f * f));
    }
}

cudaError_t hl_launch_pool(const hl_pool_img *imgs, int nimg, int side,
                           __nv_bfloat16 *out, cudaStream_t s)
{
    const size_t n = (size_t)nimg * side * side;
    const int blocks = (int)std::min((n + 255) / 256, (size_t)65536);
    hl_pool_kernel<<<std::max(blocks, 1), 256, 0, s>>>(imgs, nimg, side, out);
    return cudaGetLastError();
}

/* ---- weight gradients ------------------------------------------------------ */

/* dw[co][tap][ci] += sum over output pixels p of dy[p][co] * x[in(p, tap)][ci]:
 * a GEMM whose contraction runs over the pixels, K = 16 neighbouring pixels of
 * a row an MMA, both operands MN-major (a core matrix is 8 pixels x 8 channels,
 * the same 128 bytes as in the convolutions).
 *   A (M = 128): the x halo as rows of four channel planes; row group
 *     4 ky + q of a pixel row is plane q of the halo row ky further down, all
 *     one plane row apart, so one descriptor holds three ky x 32 channels
 *     (rows 0..95; rows 96..127 run into the row after and are not read
 *     back).  kx is a start address, with its own accumulator.
 *   B: dy, N = 32 channels -- or, for the one-channel FP32 gradient, N = 16
 *     with dy split exactly into three bf16 pieces (columns 0..2), whose sums
 *     are added at the end.
 * dy of the 32-channel layers is bf16 already, so the products are exact.  The
 * tensor cores truncate their FP32 sums, which over hundreds of additions
 * outgrows the rounding of FP32 fused multiply-adds (measured against 64 bits:
 * up to 2e-6 where those had 4e-7), so an accumulator takes DW_SEQ MMAs only
 * and is then added, rounded to nearest, to a thread's register sums (1.3e-7
 * to 4e-7, at or below the FP32 kernel's).  Bound by the copies into shared
 * memory and the MMAs' reads of A.  32 maps: 64 x 64 x 32 layers 12.8 us a
 * launch, the stride-2 layer 18, the input layer 19, the one-channel output 11,
 * where FP32 multiply-adds took 222, 222, 400 and 210. */
#define DW_SEQ 4       /* MMAs (rows of 16 pixels) an accumulator takes */
#define DW_SETS (DW_TY / DW_SEQ)
#define DW_TX 16
#define DW_TY 8
template <int STRIDE> struct DwHalo;
template <> struct DwHalo<1> {
    /* 10 rows of 18 pixels, one more row for the unused row groups */
    static constexpr int COLS = 18, ROWS = 10, P = 288, HALF = 0, BYTES = 11 * 4 * 288;
};
template <> struct DwHalo<2> {
    /* 17 rows of 33 pixels, even and odd columns apart (64 bytes off each
     * other's banks) */
    static constexpr int COLS = 33, ROWS = 17, P = 272, HALF = 18 * 4 * 272 + 64,
                         BYTES = 2 * (18 * 4 * 272 + 64);
};
#define DW_DYP 288     /* plane row of the dy tile: 16 pixels and 32 bytes of padding */

template <int XBYTES, int DYG>
struct DwSmem {
    alignas(128) unsigned char x[2][(XBYTES + 127) / 128 * 128];
    alignas(128) unsigned char dy[2][DW_TY * DYG * DW_DYP];
    unsigned long long bar;
    unsigned tmem;
};

/* D f32, A and B bf16, both MN-major */
__host__ __device__ constexpr unsigned mma_idesc_mn(int M, int N)
{
    return mma_idesc(M, N) | (1u << 15) | (1u << 16);
}

/* copies of a dy tile: 16 x 8 pixels, four planes a row, zero past the map */
__device__ __forceinline__ void dw_load_dy(const hl_dw_args &a, const ConvTile &t, unsigned dst)
{
    const int q = threadIdx.x & 3;
    for (int px = threadIdx.x >> 2; px < DW_TX * DW_TY; px += CNN_THREADS / 4) {
        const int y = px / DW_TX, x = px % DW_TX;
        const bool ok = t.y0 + y < a.Ho && t.x0 + x < a.Wo;
        const __nv_bfloat16 *src =
            ok ? a.dy + (((size_t)t.b * a.Ho + t.y0 + y) * a.Wo + t.x0 + x) * 32 + q * 8 : a.dy;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                     ::"r"(dst + (unsigned)((y * 4 + q) * DW_DYP + x * 16)), "l"(src),
                     "r"(ok ? 16 : 0)
                     : "memory");
    }
}

template <int STRIDE, bool SPLIT>
__global__ void __launch_bounds__(CNN_THREADS)
hl_dw32_kernel(hl_dw_args a)
{
    using H = DwHalo<STRIDE>;
    constexpr int DYG = SPLIT ? 2 : 4;
    constexpr int N = SPLIT ? 16 : 32;
    extern __shared__ __align__(128) unsigned char conv_raw[];
    typedef DwSmem<H::BYTES, DYG> Smem;
    Smem &sm = *reinterpret_cast<Smem *>(conv_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned tmem = conv_begin(&sm.tmem, &sm.bar, 256);
    hl_pdl_begin();
    const int tx_n = (a.Wo + DW_TX - 1) / DW_TX, ty_n = (a.Ho + DW_TY - 1) / DW_TY;
    const int ntiles = a.B * tx_n * ty_n;
    const unsigned xbase = cnn_smem_u32(sm.x[0]), dybase = cnn_smem_u32(sm.dy[0]);
    constexpr unsigned XST = sizeof(sm.x[0]), DYST = sizeof(sm.dy[0]);

    auto load = [&](const ConvTile &t, unsigned st) {
        const int iy0 = t.y0 * STRIDE - 1, ix0 = t.x0 * STRIDE - 1;
        const int q = tid & 3;
        const __nv_bfloat16 *x = a.x + (size_t)t.b * a.H * a.W * 32 + q * 8;
        int hy = (tid >> 2) / H::COLS, hx = (tid >> 2) % H::COLS;
        for (int px = tid >> 2; px < H::ROWS * H::COLS; px += CNN_THREADS / 4) {
            const int iy = iy0 + hy, ix = ix0 + hx;
            const bool ok = (unsigned)iy < (unsigned)a.H && (unsigned)ix < (unsigned)a.W;
            const __nv_bfloat16 *src = ok ? x + (size_t)(iy * a.W + ix) * 32 : a.x;
            const unsigned dst =
                xbase + st * XST + (unsigned)((hy * 4 + q) * H::P) +
                (STRIDE == 2 ? (unsigned)((hx & 1) * H::HALF + (hx >> 1) * 16)
                             : (unsigned)(hx * 16));
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                         ::"r"(dst), "l"(src), "r"(ok ? 16 : 0)
                         : "memory");
            hx += 32 % H::COLS;
            hy += 32 / H::COLS;
            if (hx >= H::COLS) {
                hx -= H::COLS;
                hy++;
            }
        }
        if (!SPLIT) {
            dw_load_dy(a, t, dybase + st * DYST);
        } else {
            /* one pixel a thread: f = hi + mid + lo exactly (24 bits in three
             * pieces of 8); an infinity or NaN stays in hi alone */
            const int y = tid / DW_TX, xx = tid % DW_TX;
            const bool ok = t.y0 + y < a.Ho && t.x0 + xx < a.Wo;
            const float f =
                ok ? a.dy_f32[((size_t)t.b * a.Ho + t.y0 + y) * a.Wo + t.x0 + xx] : 0.0f;
            const __nv_bfloat16 hi = __float2bfloat16(f);
            float r = __fsub_rn(f, __bfloat162float(hi));
            r = fabsf(f) < 3.0e38f ? r : 0.0f;
            const __nv_bfloat16 mid = __float2bfloat16(r);
            const __nv_bfloat16 lo = __float2bfloat16(__fsub_rn(r, __bfloat162float(mid)));
            unsigned char *d = sm.dy[st] + (y * 2) * DW_DYP + xx * 16;
            *reinterpret_cast<uint4 *>(d) = make_uint4(
                (unsigned)__bfloat16_as_ushort(hi) | ((unsigned)__bfloat16_as_ushort(mid) << 16),
                (unsigned)__bfloat16_as_ushort(lo), 0u, 0u);
            *reinterpret_cast<uint4 *>(d + DW_DYP) = make_uint4(0u, 0u, 0u, 0u);
        }
    };

    ConvTiles<DW_TX, DW_TY> walk(tx_n, ty_n);
    float acc[3][SPLIT ? 1 : 32];   /* warp = ky, lane = ci: this thread's sums */
#pragma unroll
    for (int kx = 0; kx < 3; kx++)
#pragma unroll
        for (int c = 0; c < (SPLIT ? 1 : 32); c++)
            acc[kx][c] = 0.0f;
    bool failed = false;
    unsigned it = 0;
    if ((int)blockIdx.x < ntiles)
        load(walk.get(), 0);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, it++) {
        const unsigned st = it & 1u;
        asm volatile("cp.async.wait_all;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (__syncthreads_or(failed))
            break;
        if (tid < 32 && elect_one()) {
            tmem_fence_after();
            const unsigned long long ad0 = smem_desc(xbase + st * XST, 128, H::P);
            const unsigned long long bd0 = smem_desc(dybase + st * DYST, 128, DW_DYP);
#pragma unroll
            for (int y = 0; y < DW_TY; y++)
#pragma unroll
                for (int kx = 0; kx < 3; kx++) {
                    const unsigned off =
                        (unsigned)(y * STRIDE * 4 * H::P) +
                        (STRIDE == 2 ? (unsigned)((kx & 1) * H::HALF + (kx >> 1) * 16)
                                     : (unsigned)(kx * 16));
                    umma_f16(tmem + (unsigned)((y / DW_SEQ * 3 + kx) * 32), ad0 + (off >> 4),
                             bd0 + (unsigned)(y * DYG * DW_DYP >> 4),
                             mma_idesc_mn(CNN_TILE_M, N), y % DW_SEQ > 0);
                }
            umma_commit(&sm.bar);
        }
        __syncwarp();
        /* the other buffer's MMAs were waited for in the round before */
        if (tile + (int)gridDim.x < ntiles) {
            walk.next();
            load(walk.get(), st ^ 1u);
        }
        if (!cnn_mbar_wait(&sm.bar, it & 1u)) {
            failed = true;
            if (lane == 0)
                atomicOr(a.status, HL_ST_CNN_TIMEOUT);
            continue;
        }
        tmem_fence_after();
        if (warp < 3) {   /* rows 32 ky + ci of every accumulator */
#pragma unroll
            for (int set = 0; set < DW_SETS; set++)
#pragma unroll
                for (int kx = 0; kx < 3; kx++) {
                    float v[32];
                    tmem_ld32(tmem + ((unsigned)(32 * warp) << 16) +
                                  (unsigned)((set * 3 + kx) * 32), v);
                    if (SPLIT) {
                        acc[kx][0] += v[0] + (v[1] + v[2]);
                    } else {
#pragma unroll
                        for (int c = 0; c < (SPLIT ? 1 : 32); c++)
                            acc[kx][c] += v[c];
                    }
                }
        }
        tmem_fence_before();
    }
    if (failed)
        cnn_mbar_wait(&sm.bar, it & 1u);   /* as in hl_conv32_kernel */
    if (!__syncthreads_or(failed) && it > 0 && warp < 3) {
#pragma unroll
        for (int kx = 0; kx < 3; kx++) {
            float *dst = a.dw + (size_t)(blockIdx.x % HL_GRAD_COPIES) * a.dw_stride +
                         (warp * 3 + kx) * 32 + lane;
#pragma unroll
            for (int c = 0; c < (SPLIT ? 1 : 32); c++)
                atomicAdd(dst + c * 288, acc[kx][c]);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    tmem_fence_before();
    __syncthreads();
    if (tid < 32)
        tmem_dealloc(tmem, 256);
}

/* One input channel (stride 1 or 2): A's rows are the 9 taps, two 8-tap
 * groups a pixel gathered by its thread; the row groups past them run into the
 * rows after (14 spare plane rows at the end) and are not read back. */
#define DW1_X ((DW_TY * 2 + 14) * DW_DYP)
__global__ void __launch_bounds__(CNN_THREADS)
hl_dw1_kernel(hl_dw_args a)
{
    extern __shared__ __align__(128) unsigned char conv_raw[];
    typedef DwSmem<DW1_X, 4> Smem;
    Smem &sm = *reinterpret_cast<Smem *>(conv_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned tmem = conv_begin(&sm.tmem, &sm.bar, 64);
    hl_pdl_begin();
    const int tx_n = (a.Wo + DW_TX - 1) / DW_TX, ty_n = (a.Ho + DW_TY - 1) / DW_TY;
    const int ntiles = a.B * tx_n * ty_n;
    const unsigned xbase = cnn_smem_u32(sm.x[0]), dybase = cnn_smem_u32(sm.dy[0]);
    constexpr unsigned XST = sizeof(sm.x[0]), DYST = sizeof(sm.dy[0]);
    const int py = tid / DW_TX, px = tid % DW_TX;   /* the thread's pixel */

    auto load = [&](const ConvTile &t, unsigned st) {
        dw_load_dy(a, t, dybase + st * DYST);
        const int iy0 = (t.y0 + py) * a.stride - 1, ix0 = (t.x0 + px) * a.stride - 1;
        const unsigned short *x =
            reinterpret_cast<const unsigned short *>(a.x) + (size_t)t.b * a.H * a.W;
        unsigned short v[9];
#pragma unroll
        for (int ky = 0; ky < 3; ky++) {
            const bool oky = (unsigned)(iy0 + ky) < (unsigned)a.H;
            const unsigned short *row = x + (ptrdiff_t)(iy0 + ky) * a.W + ix0;
#pragma unroll
            for (int kx = 0; kx < 3; kx++)
                v[3 * ky + kx] = oky && (unsigned)(ix0 + kx) < (unsigned)a.W ? row[kx]
                                                                             : (unsigned short)0;
        }
        unsigned char *d = sm.x[st] + (py * 2) * DW_DYP + px * 16;
        *reinterpret_cast<uint4 *>(d) =
            make_uint4(v[0] | ((unsigned)v[1] << 16), v[2] | ((unsigned)v[3] << 16),
                       v[4] | ((unsigned)v[5] << 16), v[6] | ((unsigned)v[7] << 16));
        *reinterpret_cast<uint4 *>(d + DW_DYP) = make_uint4(v[8], 0u, 0u, 0u);
    };

    ConvTiles<DW_TX, DW_TY> walk(tx_n, ty_n);
    float acc[32];   /* warp 0, lane = tap: this thread's sums */
#pragma unroll
    for (int c = 0; c < 32; c++)
        acc[c] = 0.0f;
    bool failed = false;
    unsigned it = 0;
    if ((int)blockIdx.x < ntiles)
        load(walk.get(), 0);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, it++) {
        const unsigned st = it & 1u;
        asm volatile("cp.async.wait_all;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (__syncthreads_or(failed))
            break;
        if (tid < 32 && elect_one()) {
            tmem_fence_after();
            const unsigned long long ad0 = smem_desc(xbase + st * XST, 128, DW_DYP);
            const unsigned long long bd0 = smem_desc(dybase + st * DYST, 128, DW_DYP);
#pragma unroll
            for (int y = 0; y < DW_TY; y++)
                umma_f16(tmem + (unsigned)(y / DW_SEQ * 32), ad0 + (unsigned)(y * 2 * DW_DYP >> 4),
                         bd0 + (unsigned)(y * 4 * DW_DYP >> 4), mma_idesc_mn(CNN_TILE_M, 32),
                         y % DW_SEQ > 0);
            umma_commit(&sm.bar);
        }
        __syncwarp();
        if (tile + (int)gridDim.x < ntiles) {
            walk.next();
            load(walk.get(), st ^ 1u);
        }
        if (!cnn_mbar_wait(&sm.bar, it & 1u)) {
            failed = true;
            if (lane == 0)
                atomicOr(a.status, HL_ST_CNN_TIMEOUT);
            continue;
        }
        tmem_fence_after();
        if (warp == 0) {
#pragma unroll
            for (int set = 0; set < DW_SETS; set++) {
                float v[32];
                tmem_ld32(tmem + (unsigned)(set * 32), v);
#pragma unroll
                for (int c = 0; c < 32; c++)
                    acc[c] += v[c];
            }
        }
        tmem_fence_before();
    }
    if (failed)
        cnn_mbar_wait(&sm.bar, it & 1u);   /* as in hl_conv32_kernel */
    if (!__syncthreads_or(failed) && it > 0 && warp == 0 && lane < 9) {
#pragma unroll
        for (int co = 0; co < 32; co++)
            atomicAdd(a.dw + (size_t)(blockIdx.x % HL_GRAD_COPIES) * a.dw_stride + co * 9 + lane,
                      acc[co]);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    tmem_fence_before();
    __syncthreads();
    if (tid < 32)
        tmem_dealloc(tmem, 64);
}

template <typename K>
static cudaError_t launch_dw(K kernel, size_t smem, int ctas_per_sm, const hl_dw_args *a,
                             cudaStream_t s)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const cudaError_t e =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess)
        return e;
    const long long nt = (long long)a->B * ((a->Wo + DW_TX - 1) / DW_TX) *
                         ((a->Ho + DW_TY - 1) / DW_TY);
    if (nt > 0x7fffffffLL)
        return cudaErrorInvalidValue;
    const int grid = (int)std::max(1LL, std::min(nt, (long long)sms * ctas_per_sm));
    return hl_launch_pdl(kernel, dim3(grid), dim3(CNN_THREADS), smem, s, false, *a);
}

cudaError_t hl_launch_conv_dw(const hl_dw_args *a, cudaStream_t s)
{
    if (a->cin == 1 && a->dy)
        return launch_dw(hl_dw1_kernel, sizeof(DwSmem<DW1_X, 4>), 3, a, s);
    if (a->cin != 32)
        return cudaErrorInvalidValue;
    if (!a->dy)
        return a->stride == 1 ? launch_dw(hl_dw32_kernel<1, true>,
                                          sizeof(DwSmem<DwHalo<1>::BYTES, 2>), 2, a, s)
                              : cudaErrorInvalidValue;
    return a->stride == 2 ? launch_dw(hl_dw32_kernel<2, false>,
                                      sizeof(DwSmem<DwHalo<2>::BYTES, 4>), 2, a, s)
                          : launch_dw(hl_dw32_kernel<1, false>,
                                      sizeof(DwSmem<DwHalo<1>::BYTES, 4>), 2, a, s);
}

/* ---- coarse Hough head ------------------------------------------------------ */

/* cos and sin of the coarse angles (t + 0.5) * pi / HL_HEAD_T, evaluated in
 * double on the host and rounded to float; passed by value */
struct HeadTrig {
    float c[HL_HEAD_T], s[HL_HEAD_T];
};

static const HeadTrig &head_trig()
{
    static const HeadTrig t = [] {   /* once, whichever thread comes first */
        HeadTrig v;
        for (int i = 0; i < HL_HEAD_T; i++) {
            const double th = ((double)i + 0.5) * 3.14159265358979323846 / HL_HEAD_T;
            v.c[i] = (float)cos(th);
            v.s[i] = (float)sin(th);
        }
        return v;
    }();
    return t;
}

/* bin of evidence cell (qy, qx) of image geometry g at coarse angle t; every
 * operation rounded as written so the CPU oracle reproduces it */
__device__ __forceinline__ int head_bin(const hl_head_geom &g, int qy, int qx,
                                        float c, float s)
{
    const float x = __fmul_rn(__fadd_rn((float)qx, 0.5f), g.cell);
    const float y = __fmul_rn(__fadd_rn((float)qy, 0.5f), g.cell);
    const float rho = __fadd_rn(__fmul_rn(x, c), __fmul_rn(y, s));
    int r = (int)floorf(__fmul_rn(__fsub_rn(rho, g.rho_min), g.inv_rw));
    return min(max(r, 0), HL_HEAD_R - 1);
}

/* logits[b][t][r] = alpha * sum_{cells with bin r at angle t} e[b][cell] + beta
 * One CTA per (image, group of HEAD_TG angles), the group's [HEAD_TG][R] sums
 * and the image's evidence map in shared memory (rows one word longer than the
 * map, so a walk along x or y is free of bank conflicts).  A thread walks one
 * line of evidence cells for one angle -- a column when the angle's rho
 * changes less along y (|sin| < |cos|), else a row -- keeping a running sum
 * while consecutive cells fall in one bin and adding it to that bin when the
 * bin changes: the cells of a line mostly share bins, so this issues a few
 * shared reductions per line instead of one per cell.  Bound by its
 * instructions and shared reductions: 64 images 30.3 us, 95 us with 64-bit
 * shared atomics and a double conversion per cell; prefix sums along the lines
 * with one difference per bin measured 38 us.  The sums are 64-bit
 * fixed point (2^-24 units), so they do not depend on the order of the
 * additions; a sum is kept in two 32-bit words (a 64-bit shared reduction is a
 * compare-and-swap loop): where every cell fits 32 bits, run = hi * 2^20 + lo
 * (at most 64 runs reach a bin, one a line, so neither word overflows and
 * neither reduction needs its result back), else low and high word with the
 * carry. */
#define HEAD_TG 6
#define HEAD_EV 64          /* side of the evidence map */
#define HEAD_FIX 16777216.0f
#define HEAD_WORDS (HEAD_TG * HL_HEAD_R + 32)   /* the bins, a dump word per lane */
__device__ __forceinline__ void head_add64(unsigned *lo, unsigned *hi, unsigned long long v)
{
    const unsigned l = (unsigned)v;
    const unsigned old = atomicAdd(lo, l);
    const unsigned h = (unsigned)(v >> 32) + (old + l < old ? 1u : 0u);
    if (h)
        atomicAdd(hi, h);
}
/* 64-bit conversions run on the FP64 pipe (16 cycles a warp even when
 * predicated off), so they are kept out of line */
static __device__ __noinline__ float head_sum64(long long fx)
{
    return (float)((double)fx * (1.0 / HEAD_FIX));
}

/* the bin of rho (head_bin) */
__device__ __forceinline__ int head_cell(float fi, float fixed, float mc, const hl_head_geom &g)
{
    /* head_bin's roundings; fl(x c) + fl(y s) does not depend on the order */
    const float rho = __fadd_rn(fixed, __fmul_rn(__fmul_rn(fi, g.cell), mc));
    const int bin = (int)floorf(__fmul_rn(__fsub_rn(rho, g.rho_min), g.inv_rw));
    return min(max(bin, 0), HL_HEAD_R - 1);
}

/* One thread's walk of a line of n cells: cell i adds s_e[i * step] to the
 * bin of rho = fixed + m(i).  At every cell each lane issues the two
 * reductions of its run, to the bin where it leaves one and to its dump word
 * elsewhere: neighbouring lines change bins at different cells, so a branch
 * would be taken at nearly every cell. */
__device__ __forceinline__ void head_walk(const int *s_e, int step, int n, float fixed, float mc,
                                          const hl_head_geom &g, unsigned lo, unsigned dump)
{
    long long run = 0;
    int cur = 0;
    float fi = 0.5f;
    auto flush = [&](bool p) {
        const unsigned addr = p ? lo + 4u * (unsigned)cur : dump;
        asm volatile("red.shared.add.u32 [%0], %1;\n\tred.shared.add.u32 [%0 + %3], %2;"
                     ::"r"(addr), "r"((unsigned)run & 0xfffffu), "r"((unsigned)(run >> 20)),
                     "n"(HEAD_WORDS * 4)
                     : "memory");
    };
#pragma unroll 4
    for (int i = 0; i < n; i++, s_e += step, fi += 1.0f) {
        const int bin = head_cell(fi, fixed, mc, g);
        const int v = *s_e;
        const bool p = bin != cur;
        flush(p);
        run = p ? (long long)v : run + v;
        cur = bin;
    }
    flush(n > 0);
}

/* the same with the evidence read from global memory, where a cell's fixed
 * point needs more than 32 bits */
__device__ __noinline__ void head_walk_wide(const float *g_e, int gstep, int n, float fixed,
                                            float mc, const hl_head_geom &g, unsigned *lo,
                                            unsigned *hi)
{
    unsigned long long run = 0ull;
    int cur = 0;
    float fi = 0.5f;
    for (int i = 0; i < n; i++, fi += 1.0f) {
        const int bin = head_cell(fi, fixed, mc, g);
        if (bin != cur) {
            head_add64(lo + cur, hi + cur, run);
            cur = bin;
            run = 0ull;
        }
        run += (unsigned long long)__float2ll_rn(g_e[i * gstep] * HEAD_FIX);
    }
    head_add64(lo + cur, hi + cur, run);
}

__global__ void __launch_bounds__(384)
hl_head_fwd_kernel(const float *e, const hl_head_geom *geo,
                   const float *ab, float *hsum, float *logits, HeadTrig tr)
{
    __shared__ unsigned s_sum[2 * HEAD_WORDS];     /* low words, high words */
    __shared__ int s_e[HEAD_EV * (HEAD_EV + 1)];   /* the evidence in fixed point */
    __shared__ float cs[HEAD_TG], sn[HEAD_TG];
    const int b = blockIdx.y, t0 = blockIdx.x * HEAD_TG;
    const int nt = min(HEAD_TG, HL_HEAD_T - t0);
    unsigned *const s_lo = s_sum, *const s_hi = s_sum + HEAD_WORDS;
    for (int i = threadIdx.x; i < 2 * HEAD_WORDS; i += blockDim.x)
        s_sum[i] = 0u;
    if (threadIdx.x < nt) {
        cs[threadIdx.x] = tr.c[t0 + threadIdx.x];
        sn[threadIdx.x] = tr.s[t0 + threadIdx.x];
    }
    hl_pdl_begin();
    const hl_head_geom g = geo[b];
    const float *eb = e + (size_t)b * HEAD_EV * HEAD_EV;
    bool big = false;   /* a value whose fixed point needs more than 32 bits */
    for (int i = threadIdx.x; i < HEAD_EV * HEAD_EV; i += blockDim.x) {
        const float x = eb[i] * HEAD_FIX;
        big |= !(fabsf(x) < 2147483648.0f);
        s_e[(i / HEAD_EV) * (HEAD_EV + 1) + i % HEAD_EV] = __float2int_rn(x);
    }
    const bool wide = __syncthreads_or(big);
    for (int job = threadIdx.x; job < nt * HEAD_EV; job += blockDim.x) {
        const int t = job / HEAD_EV, line = job % HEAD_EV;
        const float c = cs[t], sv = sn[t];
        const bool walk_y = fabsf(sv) < fabsf(c);
        /* the walk's fixed and moving coordinates */
        const int n = line < (walk_y ? g.qw : g.qh) ? min(walk_y ? g.qh : g.qw, HEAD_EV) : 0;
        const float fixed = __fmul_rn(__fmul_rn(__fadd_rn((float)line, 0.5f), g.cell),
                                      walk_y ? c : sv);
        const float mc = walk_y ? sv : c;
        const int *p = s_e + (walk_y ? line : line * (HEAD_EV + 1));
        const int step = walk_y ? HEAD_EV + 1 : 1;
        if (!wide)
            head_walk(p, step, n, fixed, mc, g, cnn_smem_u32(s_lo + t * HL_HEAD_R),
                      cnn_smem_u32(s_lo + HEAD_TG * HL_HEAD_R + (threadIdx.x & 31)));
        else
            head_walk_wide(eb + (walk_y ? line : line * HEAD_EV), walk_y ? HEAD_EV : 1, n, fixed,
                           mc, g, s_lo + t * HL_HEAD_R, s_hi + t * HL_HEAD_R);
    }
    __syncthreads();
    const float alpha = ab[0], beta = ab[1];
    for (int i = threadIdx.x; i < nt * HL_HEAD_R; i += blockDim.x) {
        const size_t o = (size_t)b * HL_HEAD_T * HL_HEAD_R + (size_t)t0 * HL_HEAD_R + i;
        const long long fx =
            wide ? (long long)(((unsigned long long)s_hi[i] << 32) | s_lo[i])
                 : (((long long)(int)s_hi[i]) << 20) + (long long)s_lo[i];
        /* the double only where the sum needs more than 32 bits: both give
         * the float nearest the sum */
        const float sum = fx == (int)fx ? __int2float_rn((int)fx) * (1.0f / HEAD_FIX)
                                        : head_sum64(fx);
        if (hsum)
            hsum[o] = sum;
        logits[o] = alpha * sum + beta;
    }
}

/* de[b][cell] = alpha * sum_t dz[b][t][bin(cell, t)] (the gather transpose of
 * the head), its bf16 copy (the next convolution's operand) and its sum (the
 * last layer's bias gradient); one CTA per (image, 512 cells), each thread one
 * cell summing its angles in order */
__global__ void __launch_bounds__(512)
hl_head_bwd_kernel(const float *dz, int ev, const hl_head_geom *geo,
                   const float *ab, float *de, __nv_bfloat16 *de_b, float *db, int db_stride,
                   HeadTrig tr)
{
    __shared__ float s_tot[16];
    __shared__ float sd[HL_HEAD_T * HL_HEAD_R];
    __shared__ float cs[HL_HEAD_T], sn[HL_HEAD_T];
    const int b = blockIdx.y;
    if (threadIdx.x < HL_HEAD_T) {
        cs[threadIdx.x] = tr.c[threadIdx.x];
        sn[threadIdx.x] = tr.s[threadIdx.x];
    }
    hl_pdl_begin();
    for (int i = threadIdx.x; i < HL_HEAD_T * HL_HEAD_R; i += blockDim.x)
        sd[i] = dz[(size_t)b * HL_HEAD_T * HL_HEAD_R + i];
    __syncthreads();
    const hl_head_geom g = geo[b];
    const float alpha = ab[0];
    float tot = 0.0f;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < ev * ev;
         p += gridDim.x * blockDim.x) {
        const int qy = p / ev, qx = p % ev;
        float acc = 0.0f;
        if (qy < g.qh && qx < g.qw)
            for (int t = 0; t < HL_HEAD_T; t++)
                acc += sd[t * HL_HEAD_R + head_bin(g, qy, qx, cs[t], sn[t])];
        const float v = alpha * acc;
        de[(size_t)b * ev * ev + p] = v;
        de_b[(size_t)b * ev * ev + p] = __float2bfloat16(v);
        tot += v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        tot += __shfl_xor_sync(FULL, tot, o);
    if ((threadIdx.x & 31) == 0)
        s_tot[threadIdx.x >> 5] = tot;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 16; w++)
            tot += s_tot[w];
        atomicAdd(db + (size_t)((blockIdx.x + blockIdx.y) % HL_GRAD_COPIES) * db_stride, tot);
    }
}

cudaError_t hl_launch_head_fwd(const float *e, const hl_head_geom *geo,
                               int nimg, const float *ab, float *hsum,
                               float *logits, cudaStream_t s)
{
    return hl_launch_pdl(hl_head_fwd_kernel, dim3((HL_HEAD_T + HEAD_TG - 1) / HEAD_TG, nimg),
                         dim3(384), 0, s, false, e, geo, ab, hsum, logits, head_trig());
}

cudaError_t hl_launch_head_bwd(const float *dz, int ev, const hl_head_geom *geo,
                               int nimg, const float *ab, float *de, __nv_bfloat16 *de_b,
                               float *db, int db_stride, cudaStream_t s)
{
    return hl_launch_pdl(hl_head_bwd_kernel, dim3((unsigned)((ev * ev + 511) / 512), nimg),
                         dim3(512), 0, s, false, dz, ev, geo, ab, de, de_b, db, db_stride,
                         head_trig());
}

/* ---- loss ------------------------------------------------------------------- */

/* Weighted binary cross-entropy on logits: per cell
 * l = -(wpos * y * log s + (1 - y) * log(1 - s)), s = sigmoid(z); dz = dl/dz /
 * n; also d alpha = sum dz * hsum, d beta = sum dz and the summed loss. */
__global__ void hl_bce_kernel(const float *z, const float *y, const float *hsum,
                              long long n, float wpos, float *dz, float *dab,
                              float *loss, int stride)
{
    __shared__ float r[3][256];
    float la = 0.0f, ga = 0.0f, gb = 0.0f;
    hl_pdl_begin();
    const float inv = 1.0f / (float)n;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n;
         e += (long long)gridDim.x * blockDim.x) {
        const float zz = z[e], yy = y[e];
        /* log(1 + exp(-|z|)) form, stable for large |z| */
        const float sp = log1pf(expf(-fabsf(zz)));
        const float log_s = fminf(zz, 0.0f) - sp;       /* log sigmoid(z) */
        const float log_1s = fminf(-zz, 0.0f) - sp;     /* log(1 - sigmoid(z)) */
        la += -(wpos * yy * log_s + (1.0f - yy) * log_1s);
        const float sg = 1.0f / (1.0f + expf(-zz));
        const float g = (wpos * yy * (sg - 1.0f) + (1.0f - yy) * sg) * inv;
        dz[e] = g;
        ga += g * hsum[e];
        gb += g;
    }
    r[0][threadIdx.x] = la;
    r[1][threadIdx.x] = ga;
    r[2][threadIdx.x] = gb;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o)
            for (int k = 0; k < 3; k++)
                r[k][threadIdx.x] += r[k][threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const size_t c = (size_t)(blockIdx.x % HL_GRAD_COPIES) * stride;
        atomicAdd(loss + c, r[0][0] * inv);
        atomicAdd(dab + c, r[1][0]);
        atomicAdd(dab + c + 1, r[2][0]);
    }
}

cudaError_t hl_launch_bce(const float *z, const float *y, const float *hsum,
                          long long n, float wpos, float *dz, float *dab,
                          float *loss, int stride, cudaStream_t s)
{
    return hl_launch_pdl(hl_bce_kernel, dim3(256), dim3(256), 0, s, false, z, y, hsum, n, wpos,
                         dz, dab, loss, stride);
}

/* ---- Adam and weight layouts ---------------------------------------------- */

/* One thread per parameter: the sum of the gradient copies, the Adam update
 * (lr > 0), then the bf16 copies of
 * a layer's FP32 master weights [cout][9 * cin]: the forward operand (same
 * layout) and, past the first layer, the backward one -- stride 1: flipped and
 * transposed ([cin][8 - tap][cout], the input gradient as a convolution),
 * stride 2: transposed ([cin][tap][cout], the input-gradient gather). */
__global__ void hl_update_kernel(hl_update_args a)
{
    hl_pdl_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n)
        return;
    if (a.gsum) {   /* a step: the copies' gradient (and, last, the loss) */
        float gs = 0.0f;
#pragma unroll
        for (int c = 0; c < HL_GRAD_COPIES; c++)
            gs += a.gpart[(size_t)c * a.gstride + i];
        a.g[i] = gs;
        if (i == 0) {
            float ls = 0.0f;
#pragma unroll
            for (int c = 0; c < HL_GRAD_COPIES; c++)
                ls += a.gpart[(size_t)c * a.gstride + a.n];
            a.g[a.n] = ls;
        }
    }
    float w = a.w[i];
    if (a.lr > 0.0f) {
        const float b1 = 0.9f, b2 = 0.999f;
        const float gi = fminf(fmaxf(a.g[i], -a.clip), a.clip);
        const float mi = b1 * a.m[i] + (1.0f - b1) * gi;
        const float vi = b2 * a.v[i] + (1.0f - b2) * gi * gi;
        a.m[i] = mi;
        a.v[i] = vi;
        w -= a.lr * (mi * a.c1) / (sqrtf(vi * a.c2) + 1e-8f);
        a.w[i] = w;
    }
    for (int l = 0; l < a.nlayers; l++) {
        const hl_update_layer &L = a.layer[l];
        const int r = i - L.off;
        if (r < 0 || r >= L.cout * 9 * L.cin)
            continue;
        const __nv_bfloat16 v = __float2bfloat16(w);
        L.wf[r] = v;
        if (L.wb) {
            const int co = r / (9 * L.cin), k = r % (9 * L.cin);
            const int tap = k / L.cin, ci = k % L.cin;
            L.wb[((size_t)ci * 9 + (L.flip ? 8 - tap : tap)) * L.cout + co] = v;
        }
    }
}

cudaError_t hl_launch_update(hl_update_args *a, int step, cudaStream_t s)
{
    a->c1 = 1.0f / (1.0f - powf(0.9f, (float)step));
    a->c2 = 1.0f / (1.0f - powf(0.999f, (float)step));
    return hl_launch_pdl(hl_update_kernel, dim3((a->n + 255) / 256), dim3(256), 0, s, false, *a);
}
