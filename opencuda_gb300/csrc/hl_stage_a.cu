/*
 * hl_stage_a.cu -- cos/sin table and stage (a): edge-pixel compaction.
 *
 * Compaction replaces the flag / ScanArray / scatter chain of
 * ImgConvert::imgConvertToCst (okano_3_0/ImgConvert.cu:142-353,
 * okano_3_0/ScanArray.cu:1351+) with ONE pass over the image: tiles of 128 x 32
 * pixels are read with 16-byte loads, their 255-pixels counted, the counts
 * published, the predecessors' summed and the coordinates written, by
 * persistent CTAs that pipeline groups of four tiles (batches, images of more
 * than 20 M pixels) or by one large CTA per SM (single images).  The predicate
 * is the vote kernel's `pixel == 255` (okano_3_0/HoughLine.cu:125), not
 * ImgConvert's `>= 128`.
 */
#include <algorithm>

#include "hl_internal.h"
#include "hl_device.cuh"

#define FULL 0xffffffffu

/* theta_k = (float)(k * detheta) and CUDA's cosf/sinf of it: the values the
 * reference vote kernel computes inline (okano_3_0/HoughLine.cu:115-119). */
__global__ void hl_trig_kernel(float *cosv, float *sinv, int T, int Tp,
                               double detheta)
{
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= Tp)
        return;
    if (k < T) {
        float th = (float)(k * detheta);
        cosv[k] = cosf(th);
        sinv[k] = sinf(th);
    } else {
        cosv[k] = 0.0f;
        sinv[k] = 0.0f;
    }
}

cudaError_t hl_launch_trig(float *cosv, float *sinv, int T, int Tp,
                           double detheta, cudaStream_t s)
{
    hl_trig_kernel<<<(Tp + 127) / 128, 128, 0, s>>>(cosv, sinv, T, Tp, detheta);
    return cudaGetLastError();
}

/* Look-back state word: epoch (30 bits) | flag (2 bits) | value (32 bits).
 * flag 1 = aggregate of this tile only, 2 = inclusive prefix. */
#define LB_AGG 1ull
#define LB_PRE 2ull
#define LB_SPIN_LIMIT (1 << 18)

__device__ __forceinline__ unsigned long long lb_pack(unsigned epoch,
                                                      unsigned long long flag,
                                                      unsigned value)
{
    return ((unsigned long long)epoch << 34) | (flag << 32) | value;
}

__device__ __forceinline__ void lb_store(unsigned long long *p,
                                         unsigned long long v)
{
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v)
                 : "memory");
}

__device__ __forceinline__ unsigned long long lb_load(
    const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];"
                 : "=l"(v)
                 : "l"(p)
                 : "memory");
    return v;
}

/* Warp-wide decoupled look-back (all 32 lanes of warp 0 call it) of a tile
 * whose own total is published already (as a prefix when it is the first).
 * Returns the exclusive prefix of `tile`.  Waits are bounded: past LB_SPIN_LIMIT
 * polls the status word gets HL_ST_LOOKBACK_TIMEOUT and the partial sum is
 * used, so the kernel always ends. */
__device__ int lookback(unsigned long long *state, int tile, int total,
                        unsigned epoch, int *status)
{
    const int lane = threadIdx.x & 31;
    if (tile == 0)
        return 0;
    int excl = 0;
    int top = tile - 1;
    int spins = 0;
    while (true) {
        int j = top - lane;
        unsigned long long s = 0;
        unsigned flag;
        if (j >= 0) {
            s = lb_load(&state[j]);
            flag = ((unsigned)(s >> 34) == epoch) ? (unsigned)((s >> 32) & 3u) : 0u;
        } else {
            flag = (unsigned)LB_PRE;   /* before tile 0: prefix 0 */
            s = 0;
        }
        unsigned pmask = __ballot_sync(FULL, flag == LB_PRE);
        unsigned inval = __ballot_sync(FULL, flag == 0);
        int firstp = pmask ? __ffs(pmask) - 1 : 32;
        unsigned need = (firstp >= 31) ? FULL : ((2u << firstp) - 1u);
        if (inval & need) {
            /* give up after LB_SPIN_LIMIT polls, or at once when another
             * tile already gave up, so a failure never cascades into a long
             * chain of timed-out waits */
            bool quit = ++spins > LB_SPIN_LIMIT;
            if (!quit && (spins & 255) == 0)
                quit = (*(volatile int *)status & HL_ST_LOOKBACK_TIMEOUT) != 0;
            quit = __shfl_sync(FULL, quit, 0);
            if (quit) {
                if (lane == 0)
                    atomicOr(status, HL_ST_LOOKBACK_TIMEOUT);
                break;
            }
            __nanosleep(64);
            continue;
        }
        int v = (lane <= firstp && j >= 0) ? (int)(unsigned)(s & 0xffffffffu) : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            v += __shfl_xor_sync(FULL, v, o);
        excl += v;
        if (firstp < 32)
            break;
        top -= 32;
    }
    if (lane == 0)
        lb_store(&state[tile], lb_pack(epoch, LB_PRE, (unsigned)(excl + total)));
    return excl;
}

/* Groups a launch may have for the all-predecessor prefix (below). */
#define LB_FULL_MAX 2048

/* Exclusive prefix of group g as the plain sum of every predecessor's own
 * count (all threads of the CTA call it; each group publishes only its count,
 * flag AGG, and never an inclusive prefix): a group waits just for its slowest
 * predecessor to publish, and 256 threads read up to 1024 predecessors in one
 * round trip, where the chained look-back forwards inclusive prefixes only 32
 * groups per memory round trip.  Waits are bounded as in lookback(). */
template <int NT>
__device__ int prefix_all(const unsigned long long *state, int g, unsigned epoch,
                          int *status, int *s_red)
{
    const int tid = threadIdx.x;
    int spins = 0;
    while (true) {
        int sum = 0;
        bool bad = false;
        if (g <= NT) {
            if (tid < g) {
                const unsigned long long st = lb_load(&state[tid]);
                bad = (unsigned)(st >> 34) != epoch || ((st >> 32) & 3u) == 0u;
                sum = (int)(unsigned)st;
            }
        } else for (int j0 = 0; j0 < g; j0 += 4 * NT) {
            unsigned long long st[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int j = j0 + u * NT + tid;
                st[u] = (j < g) ? lb_load(&state[j]) : 0ull;
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int j = j0 + u * NT + tid;
                if (j < g) {
                    if ((unsigned)(st[u] >> 34) != epoch || ((st[u] >> 32) & 3u) == 0u)
                        bad = true;
                    else
                        sum += (int)(unsigned)(st[u] & 0xffffffffu);
                }
            }
        }
        sum = __reduce_add_sync(FULL, sum);
        if ((tid & 31) == 0)
            s_red[tid >> 5] = sum;
        if (!__syncthreads_or(bad)) {
            int t = 0;
#pragma unroll
            for (int w = 0; w < NT / 32; w++)
                t += s_red[w];
            return t;
        }
        bool quit = ++spins > LB_SPIN_LIMIT;
        if (!quit && (spins & 255) == 0)
            quit = (*(volatile int *)status & HL_ST_LOOKBACK_TIMEOUT) != 0;
        if (__syncthreads_or(quit)) {
            if (tid == 0)
                atomicOr(status, HL_ST_LOOKBACK_TIMEOUT);
            return 0;
        }
        __nanosleep(64);
    }
}

/* A group of CT_GROUP consecutive tiles, four 16-byte loads a thread. */
#define CT_GROUP HL_COMPACT_GROUP
#define CT_CTAS_PER_SM 5
#define CT_PAD 0xffffu

struct CompactGroup {
    hl_compact_img im;
    int g;                        /* group in the batch, or -1: no more */
    int whole;                    /* four whole tiles of 16-byte aligned rows */
    int x0[CT_GROUP], y0[CT_GROUP];
    const uint8_t *p[CT_GROUP];   /* the tiles' first pixels */
};

/* Compaction of many groups (batches; images too large for the cooperative
 * kernel below) by persistent CTAs, two groups in flight each: while the
 * counts of group i are published, the image bytes of group i + 1 are on their
 * way and group i - 1, whose predecessors have had a stage's time to publish,
 * gets its prefix and is scattered.  A ticket orders the groups, so a group
 * waits only for groups that were taken before it: of the unpublished ones the
 * first never waits for another, and every wait ends.  Tickets, image numbers
 * and image records are fetched two to four groups ahead by one warp, a hop a
 * stage.
 * The points go through shared memory, so that the divergent loop over mask
 * bits is short and the list is written in whole lines.
 * 256 images, 340 MB: 137 us (243 us with a CTA a group: ticket, records, bytes,
 * prefix and scatter in one chain of 13 us, the bytes on their way for a tenth
 * of it).  Bound by instruction issue (about two thirds of the slots) and the
 * barriers of a stage; 4, 5 and 6 CTAs an SM 1095, 1097, 1109 us for the whole
 * batch call. */
__global__ void __launch_bounds__(HL_COMPACT_THREADS, CT_CTAS_PER_SM)
hl_compact_kernel(hl_compact_args a)
{
    constexpr int NW = HL_COMPACT_THREADS / 32;
    __shared__ CompactGroup s_grp[4];             /* group i in slot i & 3 */
    /* group i - 1's points: tile << 12 | row << 7 | column; CT_PAD: a sentinel */
    __shared__ unsigned short s_out[CT_GROUP * (HL_TILE_W * HL_TILE_H + 1)];
    __shared__ unsigned long long s_wsum[2][NW];  /* warps' counts, then offsets */
    __shared__ int s_tb[2][CT_GROUP + 1];         /* tile bases in the group */
    __shared__ int s_cnt[2][CT_GROUP];            /* tile counts */
    __shared__ int s_red[NW];
    __shared__ int s_excl;
    /* the fetching warp's: tickets of the slots i + 2 and i + 3, i + 2's image */
    __shared__ int s_t2, s_t3, s_i2;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ngroups = a.imgs ? a.ngroups : (a.ntiles + CT_GROUP - 1) / CT_GROUP;
    const int pad = a.pts_f2 ? 1 : 0;
    hl_pdl_begin();

    const bool fetch = warp == NW - 1;
    const auto ticket = [&](int prev) {
        int t = -1;
        if (prev >= 0 && lane == 0) {
            t = (int)(atomicAdd(a.ticket, 1u) - a.ticket_base);
            if (t >= ngroups)
                t = -1;
        }
        return t;   /* lane 0's */
    };
    const auto image_of = [&](int t) { return a.imgs && lane == 0 && t >= 0 ? a.group_img[t] : 0; };
    /* the record's words, a lane each */
    const auto record = [&](int gi) {
        gi = __shfl_sync(FULL, gi, 0);   /* lane 0's */
        return a.imgs && lane < (int)(sizeof(hl_compact_img) / 4)
                   ? reinterpret_cast<const int *>(a.imgs + gi)[lane]
                   : 0;
    };
    const auto publish_slot = [&](int slot, int t, int word) {
        CompactGroup &s = s_grp[slot];
        if (a.imgs) {
            if (lane < (int)(sizeof(hl_compact_img) / 4))
                reinterpret_cast<int *>(&s.im)[lane] = word;
        } else if (lane == 0) {
            s.im.roi = a.roi;
            s.im.tiles_x = a.tiles_x;
            s.im.ntiles = a.ntiles;
            s.im.tile_base = 0;
            s.im.group_base = 0;
            s.im.ngroups = ngroups;
            s.im.pts_base = 0;
        }
        t = __shfl_sync(FULL, t, 0);     /* lane 0's */
        __syncwarp();
        bool in = true;
        if (lane < CT_GROUP && t >= 0) {
            const int tile = (t - s.im.group_base) * CT_GROUP + lane;
            const int ty = tile / s.im.tiles_x;
            const int x = (tile - ty * s.im.tiles_x) * HL_TILE_W;
            /* tiles past the last one lie below the image */
            const int y = tile < s.im.ntiles ? ty * HL_TILE_H : s.im.roi.h;
            const uint8_t *p = s.im.roi.base + (size_t)y * (size_t)s.im.roi.pitch + x;
            s.x0[lane] = x;
            s.y0[lane] = y;
            s.p[lane] = p;
            in = y + HL_TILE_H <= s.im.roi.h && x + HL_TILE_W <= s.im.roi.w &&
                 (((uintptr_t)p | (uintptr_t)s.im.roi.pitch) & 15u) == 0;
        }
        in = __all_sync(FULL, in);
        if (lane == 0) {
            s.g = t;
            s.whole = in;
        }
    };
    if (fetch) {
        /* one ticket after the other: a CTA that took several at once would
         * hold groups that the next CTAs' first ones wait for */
        const int t0 = ticket(0);
        const int i0 = image_of(t0), t1 = ticket(t0);
        const int w0 = record(i0), i1 = image_of(t1), t2 = ticket(t1);
        publish_slot(0, t0, w0);
        const int w1 = record(i1), i2 = image_of(t2), t3 = ticket(t2);
        publish_slot(1, t1, w1);
        if (lane == 0) {
            s_t2 = t2;
            s_t3 = t3;
            s_i2 = i2;
        }
    }
    __syncthreads();

    const int r = tid >> 3, ch = tid & 7;
    /* this thread's 16 pixels of tile q: row y0 + r, columns x0 + 16 ch .. + 15 */
    uint4 v[CT_GROUP];
    const auto load = [&](const CompactGroup &s) {
        const size_t off = (size_t)r * (size_t)s.im.roi.pitch + ch * 16;
        if (s.whole) {
#pragma unroll
            for (int q = 0; q < CT_GROUP; q++)
                v[q] = __ldcs(reinterpret_cast<const uint4 *>(s.p[q] + off));
            return;
        }
#pragma unroll
        for (int q = 0; q < CT_GROUP; q++) {
            const int x = s.x0[q] + ch * 16, y = s.y0[q] + r;
            const uint8_t *p = s.p[q] + off;
            const bool vec = y < s.im.roi.h && x + 16 <= s.im.roi.w && (((uintptr_t)p) & 15u) == 0;
            v[q] = vec ? __ldcs(reinterpret_cast<const uint4 *>(p)) : make_uint4(0, 0, 0, 0);
        }
    };
    if (s_grp[0].g >= 0)
        load(s_grp[0]);
    uint32_t pm[CT_GROUP / 2] = {0u, 0u};   /* group i - 1: masks, offsets in the warp */
    unsigned long long pex = 0;
    for (int i = 0;; i++) {
        const CompactGroup &cur = s_grp[i & 3];
        const bool have = cur.g >= 0;
        const int par = i & 1;
        /* fetches for the slots i + 2 .. i + 4 */
        int w2 = 0, i3 = 0, t4 = -1;
        if (fetch) {
            w2 = record(s_i2);
            i3 = image_of(s_t3);
            t4 = ticket(s_t3);
        }
        uint32_t m[CT_GROUP / 2] = {0u, 0u};
        unsigned long long ex = 0;
        if (have) {
            unsigned long long cnt4 = 0;   /* four 16-bit counts, tile q in bits 16q */
#pragma unroll
            for (int q = 0; q < CT_GROUP; q++) {
                uint32_t mm = ff_mask16(v[q]);
                if (!cur.whole) {
                    const int x = cur.x0[q] + ch * 16;
                    if (cur.y0[q] + r < cur.im.roi.h && x < cur.im.roi.w) {
                        const uint8_t *p = cur.p[q] + (size_t)r * (size_t)cur.im.roi.pitch + ch * 16;
                        if (x + 16 > cur.im.roi.w || (((uintptr_t)p) & 15u) != 0) {
                            const int lim = min(16, cur.im.roi.w - x);
                            for (int b = 0; b < lim; b++)
                                mm |= (uint32_t)(p[b] == 255) << b;
                        }
                    }
                }
                m[q >> 1] |= mm << (16 * (q & 1));
                cnt4 |= (unsigned long long)__popc(mm) << (16 * q);
            }
            /* warp scan of the packed counts (no field exceeds 4096) */
            unsigned long long incl = cnt4;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long t = __shfl_up_sync(FULL, incl, o);
                if (lane >= o)
                    incl += t;
            }
            ex = incl - cnt4;
            if (lane == 31)
                s_wsum[par][warp] = incl;
        }
        const CompactGroup &nxt = s_grp[(i + 1) & 3];
        if (have && nxt.g >= 0)
            load(nxt);
        __syncthreads();
        if (have && warp == 0) {
            const unsigned long long ws = lane < NW ? s_wsum[par][lane] : 0ull;
            unsigned long long wi = ws;
#pragma unroll
            for (int o = 1; o < NW; o <<= 1) {
                const unsigned long long t = __shfl_up_sync(FULL, wi, o);
                if (lane >= o)
                    wi += t;
            }
            const unsigned long long tot4 = __shfl_sync(FULL, wi, NW - 1);
            if (lane < NW)
                s_wsum[par][lane] = wi - ws;
            if (lane == 0) {
                /* float2 output: every tile holds an even number of entries
                 * (one sentinel pads an odd count), so runs of tiles start and
                 * end on 16-byte boundaries */
                int run = 0;
#pragma unroll
                for (int q = 0; q < CT_GROUP; q++) {
                    const int cq = (int)((tot4 >> (16 * q)) & 0xffffu);
                    s_tb[par][q] = run;
                    s_cnt[par][q] = cq;
                    run += cq + (cq & pad);
                }
                s_tb[par][CT_GROUP] = run;
                /* the prefix runs over the image's own groups; the chained one
                 * starts from the first group's */
                const int grp = cur.g - cur.im.group_base;
                const bool first = grp == 0 && cur.im.ngroups > LB_FULL_MAX;
                lb_store(a.tile_state + cur.g, lb_pack(a.epoch, first ? LB_PRE : LB_AGG,
                                                       (unsigned)run));
            }
        }
        if (fetch) {
            publish_slot((i + 2) & 3, s_t2, w2);
            if (lane == 0) {
                s_t2 = s_t3;
                s_t3 = t4;
                s_i2 = i3;
            }
            __syncwarp();
        }
        if (i == 0) {
            __syncthreads();
        } else {
            /* group i - 1: prefix and scatter */
            const CompactGroup &pr = s_grp[(i - 1) & 3];
            const int pp = par ^ 1;
            const int grp = pr.g - pr.im.group_base;
            /* the points' places in the group, two tiles' 32 pixels at a time:
             * a tile's first place less the thread's points before it, in 16
             * bits (a tile's base counts them), plus the point's number */
            {
                unsigned long long e4 = s_wsum[pp][warp] + pex;
                int before = 0;
#pragma unroll
                for (int q = 0; q < CT_GROUP; q++) {
                    e4 += (unsigned long long)(s_tb[pp][q] - before) << (16 * q);
                    before += __popc((pm[q >> 1] >> (16 * (q & 1))) & 0xffffu);
                }
                int n = 0;
#pragma unroll
                for (int hf = 0; hf < CT_GROUP / 2; hf++) {
                    const unsigned e2 = (unsigned)(e4 >> (32 * hf));
                    const unsigned code = ((2u * hf) << 12) | (unsigned)(r << 7) | (unsigned)(ch * 16);
                    for (uint32_t mm = pm[hf]; mm; mm &= mm - 1, n++) {
                        const unsigned b = (unsigned)__ffs(mm) - 1u;
                        /* bit 4 of b is the tile: from there to bit 12 */
                        s_out[((e2 >> (b & 16u)) & 0xffffu) + n] =
                            (unsigned short)(code + b + (b & 16u) * 255u);
                    }
                }
                /* the sentinel (+infinity, 0) of an odd tile never votes inside
                 * an accumulator: its rho is infinity * cos(theta_k), and cosf
                 * of a float angle is never 0 */
                if (pad && tid < CT_GROUP && (s_cnt[pp][tid] & 1))
                    s_out[s_tb[pp][tid] + s_cnt[pp][tid]] = CT_PAD;
            }
            unsigned long long *st = a.tile_state + pr.im.group_base;
            int excl;
            if (pr.im.ngroups <= LB_FULL_MAX) {
                excl = prefix_all<HL_COMPACT_THREADS>(st, grp, a.epoch, a.status, s_red);
            } else {
                if (warp == 0) {
                    const int e = lookback(st, grp, s_tb[pp][CT_GROUP], a.epoch, a.status);
                    if (lane == 0)
                        s_excl = e;
                }
                __syncthreads();
                excl = s_excl;
            }
            if (tid < CT_GROUP) {
                const int tile = grp * CT_GROUP + tid;
                if (tile < pr.im.ntiles)
                    a.tile_off[pr.im.tile_base + tile] = excl + s_tb[pp][tid];
            } else if (tid == CT_GROUP) {
                /* the image's end (equal to the next image's start) */
                const int end = excl + s_tb[pp][CT_GROUP];
                if (grp == pr.im.ngroups - 1)
                    a.tile_off[pr.im.tile_base + pr.im.ntiles] = end;
                if (pr.g == ngroups - 1)
                    *a.count = end;
            }
            /* the points, in order, as the group's stretch of the list */
            const long long first = pr.im.pts_base + excl;
            for (int j = tid; j < s_tb[pp][CT_GROUP]; j += HL_COMPACT_THREADS) {
                const unsigned e = s_out[j], q = e >> 12;
                const unsigned x = (e & 127u) + pr.x0[q & 3], y = ((e >> 7) & 31u) + pr.y0[q & 3];
                if (!a.pts_f2)
                    a.pts[first + j] = x | (y << 16);
                else if (e == CT_PAD)
                    a.pts_f2[first + j] = make_float2(__int_as_float(0x7f800000), 0.0f);
                else
                    a.pts_f2[first + j] = make_float2((float)x, (float)y);
            }
        }
        if (!have)
            break;
#pragma unroll
        for (int q = 0; q < CT_GROUP / 2; q++)
            pm[q] = m[q];
        pex = ex;
    }
}

/* Single-image compaction with few, large CTAs: CTA c of nct takes tiles [ntiles c / nct, ntiles (c + 1) / nct) -- at most CP_MAXT --
 * with every one of its 16-byte loads in flight at once, in row order across
 * its tiles; turns them into 16-bit masks of 255-pixels in tile-major order
 * (chunk u = tile * 256 + row * 8 + column chunk, via shared memory), ranks
 * them with one block scan (a thread owns one 128-pixel row of a tile),
 * publishes one count, meets the other CTAs at one grid barrier (a
 * cooperative launch: all CTAs resident) and sums its predecessors' counts
 * in one read -- no polling of every predecessor, whose traffic grows with
 * the square of the CTA count -- then scatters one 16-pixel chunk per
 * thread.  Output as hl_compact_kernel:
 * tile-major, raster order inside a tile, odd float2 tiles padded. */
#define CP_THREADS 1024
#define CP_MAXT 32
#define CP_K (CP_MAXT * 256 / CP_THREADS)

/* tile range of CTA c of nct and the divisor of its row-order load index */
struct CpRange {
    int t0, nt, nu;
    unsigned rowlen, magic;
};
__device__ __forceinline__ CpRange cp_range(const hl_compact_args &a, int c, int nct)
{
    CpRange r;
    r.t0 = (int)((long long)a.ntiles * c / nct);
    r.nt = (int)((long long)a.ntiles * (c + 1) / nct) - r.t0;
    r.nu = r.nt * 256;
    r.rowlen = 8u * (unsigned)r.nt;
    r.magic = 0xffffffffu / r.rowlen + 1u;
    return r;
}

__global__ void __launch_bounds__(CP_THREADS, 1)
hl_compact_persist_kernel(hl_compact_args a, int nct)
{
    __shared__ int s_wsum[CP_THREADS / 32];
    __shared__ int s_tstart[CP_MAXT + 1];   /* point rank at each tile start */
    __shared__ int s_tbase[CP_MAXT];        /* tile offsets within the CTA */
    __shared__ int s_x0[CP_MAXT], s_y0[CP_MAXT];
    __shared__ int s_total, s_excl;
    __shared__ int s_red[CP_THREADS / 32];
    __shared__ __align__(16) unsigned short s_mask[CP_MAXT * 256];
    __shared__ unsigned short s_rowrel[CP_MAXT * 32];   /* row start in its tile */
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    hl_pdl_begin();
    /* a cooperative launch: every CTA is resident, so the CTA index orders
     * the prefix and the grid barrier below always completes */
    const int c = blockIdx.x;
    const CpRange R = cp_range(a, c, nct);
    const int nt = R.nt, nu = R.nu;
    if (tid < nt) {
        s_x0[tid] = ((R.t0 + tid) % a.tiles_x) * HL_TILE_W;
        s_y0[tid] = ((R.t0 + tid) / a.tiles_x) * HL_TILE_H;
    }
    __syncthreads();

    /* loads in row order across the CTA's tiles (load index L = r * 8 nt +
     * tile * 8 + column chunk: a warp reads 512 contiguous bytes of a row),
     * all in flight before any is used; r = L / (8 nt) by a multiply-high,
     * exact for L * 8 nt < 2^32 */
    uint4 v[CP_K];
#pragma unroll
    for (int k = 0; k < CP_K; k++) {
        v[k] = make_uint4(0, 0, 0, 0);
        const int L = tid + k * CP_THREADS;
        if (L < nu) {
            const int r = (int)__umulhi((unsigned)L, R.magic);
            const int rem = L - r * (int)R.rowlen;
            const int x = s_x0[rem >> 3] + (rem & 7) * 16;
            const int y = s_y0[rem >> 3] + r;
            const uint8_t *p = a.roi.base + (size_t)y * (size_t)a.roi.pitch + x;
            if (y < a.roi.h && x + 16 <= a.roi.w && (((uintptr_t)p) & 15u) == 0)
                v[k] = __ldcs((const uint4 *)p);
        }
    }
    /* 16-bit masks of 255-pixels, handed to the tile-major order through
     * shared memory (chunk u = tile * 256 + r * 8 + column chunk) */
#pragma unroll
    for (int k = 0; k < CP_K; k++) {
        const int L = tid + k * CP_THREADS;
        if (L < nu) {
            const int r = (int)__umulhi((unsigned)L, R.magic);
            const int rem = L - r * (int)R.rowlen;
            const int tl = rem >> 3, ch = rem & 7;
            const int x = s_x0[tl] + ch * 16;
            const int y = s_y0[tl] + r;
            uint32_t mm = 0;
            if (y < a.roi.h && x < a.roi.w) {
                const uint8_t *p = a.roi.base + (size_t)y * (size_t)a.roi.pitch + x;
                if (x + 16 <= a.roi.w && (((uintptr_t)p) & 15u) == 0) {
                    mm = ff_mask16(v[k]);
                } else {
                    const int lim = min(16, a.roi.w - x);
                    for (int i = 0; i < lim; i++)
                        mm |= (uint32_t)(p[i] == 255) << i;
                }
            }
            s_mask[tl * 256 + r * 8 + ch] = (unsigned short)mm;
        }
    }
    __syncthreads();
    /* ranks in tile-major order: thread tid owns row tid % 32 of tile
     * tid / 32 (chunks 8 tid .. 8 tid + 7, one 16-byte shared load); one
     * block scan of the rows' counts */
    const bool owner = tid * 8 < nu;
    int cnt = 0;
    if (owner) {
        const uint4 q = reinterpret_cast<const uint4 *>(s_mask)[tid];
        cnt = __popc(q.x) + __popc(q.y) + __popc(q.z) + __popc(q.w);
    }
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(FULL, incl, o);
        if (lane >= o)
            incl += t;
    }
    if (lane == 31)
        s_wsum[warp] = incl;
    __syncthreads();
    {
        const int ws = s_wsum[lane];
        int wi = ws;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(FULL, wi, o);
            if (lane >= o)
                wi += t;
        }
        incl += __shfl_sync(FULL, wi - ws, warp);   /* block-inclusive */
        if (tid == CP_THREADS - 1)
            s_tstart[nt] = incl;
    }
    const int base = incl - cnt;   /* rank of this row's first point */
    if (owner && (tid & 31) == 0)
        s_tstart[tid >> 5] = base;
    __syncthreads();
    if (owner)
        s_rowrel[tid] = (unsigned short)(base - s_tstart[tid >> 5]);
    /* tile offsets within the CTA (float2 output pads odd tiles); the CTA's
     * count is published, then one grid barrier (an arrival counter on the
     * ticket word, bounded spin) and one read of the predecessors' counts */
    const int pad = a.pts_f2 ? 1 : 0;
    if (warp == 0) {
        int cq = 0;
        if (lane < nt)
            cq = s_tstart[lane + 1] - s_tstart[lane];
        const int pq = cq + (cq & pad);
        int ti = pq;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(FULL, ti, o);
            if (lane >= o)
                ti += t;
        }
        if (lane < nt)
            s_tbase[lane] = ti - pq;
        const int total = __shfl_sync(FULL, ti, 31);
        if (lane == 0) {
            s_total = total;
            lb_store(&a.tile_state[c], lb_pack(a.epoch, LB_AGG, (unsigned)total));
            __threadfence();
            atomicAdd(a.ticket, 1u);
            const unsigned target = a.ticket_base + (unsigned)nct;
            int spins = 0;
            while ((int)(*(volatile unsigned *)a.ticket - target) < 0) {
                if (++spins > LB_SPIN_LIMIT) {
                    atomicOr(a.status, HL_ST_LOOKBACK_TIMEOUT);
                    break;
                }
                __nanosleep(32);
            }
            __threadfence();
        }
    }
    __syncthreads();
    {
        int sum = 0;
        for (int j = tid; j < c; j += CP_THREADS)
            sum += (int)(unsigned)(lb_load(&a.tile_state[j]) & 0xffffffffu);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            sum += __shfl_xor_sync(FULL, sum, o);
        if (lane == 0)
            s_red[warp] = sum;
        __syncthreads();
        if (tid == 0) {
            int t = 0;
            for (int w = 0; w < CP_THREADS / 32; w++)
                t += s_red[w];
            s_excl = t;
        }
        __syncthreads();
    }
    const int excl = s_excl;
    if (tid < nt)
        a.tile_off[R.t0 + tid] = excl + s_tbase[tid];
    if (c == nct - 1 && tid == 0) {
        a.tile_off[a.ntiles] = excl + s_total;
        *a.count = excl + s_total;
    }
    /* scatter, one 16-pixel chunk per thread and round (chunk u = tid +
     * 1024 k): its rank is its row's start plus the points of the row's
     * chunks before it */
#pragma unroll
    for (int k = 0; k < CP_K; k++) {
        const int u = tid + k * CP_THREADS;
        if (u >= nu)
            break;
        uint32_t mm = s_mask[u];
        if (!mm)
            continue;
        const int row = u >> 3, ch = u & 7, tl = u >> 8;
        const uint4 q = reinterpret_cast<const uint4 *>(s_mask)[row];
        const unsigned long long lo = (unsigned long long)q.x | ((unsigned long long)q.y << 32);
        const unsigned long long hi = (unsigned long long)q.z | ((unsigned long long)q.w << 32);
        const int nb = 16 * ch;
        const int before = nb >= 64 ? __popcll(lo) + __popcll(hi & ((1ull << (nb - 64)) - 1ull))
                                    : __popcll(lo & ((1ull << nb) - 1ull));
        int pos = excl + s_tbase[tl] + s_rowrel[row] + before;
        const int x = s_x0[tl] + 16 * ch;
        const int y = s_y0[tl] + (row & 31);
        while (mm) {
            const int bb = __ffs(mm) - 1;
            mm &= mm - 1;
            if (a.pts_f2)
                a.pts_f2[pos] = make_float2((float)(x + bb), (float)y);
            else
                a.pts[pos] = (uint32_t)(x + bb) | ((uint32_t)y << 16);
            pos++;
        }
    }
    /* the sentinel (+infinity, 0) of an odd float2 tile never votes inside an
     * accumulator (see hl_compact_kernel) */
    if (pad && tid < nt) {
        const int cq = s_tstart[tid + 1] - s_tstart[tid];
        if (cq & 1)
            a.pts_f2[excl + s_tbase[tid] + cq] = make_float2(__int_as_float(0x7f800000), 0.0f);
    }
}

/* CTAs of the single-image compaction: about one per SM, at most CP_MAXT
 * tiles each; 0 when that needs more CTAs than can be resident at once
 * (callers then use hl_launch_compact) */
int hl_compact_persist_ctas(int ntiles, int sms)
{
    const int need = (ntiles + CP_MAXT - 1) / CP_MAXT;
    const int nct = std::max(1, std::min(ntiles, std::max(sms, need)));
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, hl_compact_persist_kernel,
                                                      CP_THREADS, 0) != cudaSuccess)
        return 0;
    return nct <= per_sm * sms ? nct : 0;
}

cudaError_t hl_launch_compact_persist(const hl_compact_args *a, int nct, cudaStream_t s)
{
    return hl_launch_pdl(hl_compact_persist_kernel, dim3(nct), dim3(CP_THREADS), 0, s, true,
                         *a, nct);
}

static int compact_ctas(int ngroups)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::max(1, std::min(ngroups, std::max(sms, 1) * CT_CTAS_PER_SM));
}

cudaError_t hl_launch_compact(const hl_compact_args *a, cudaStream_t s)
{
    const int ngroups = a->imgs ? a->ngroups : (a->ntiles + CT_GROUP - 1) / CT_GROUP;
    return hl_launch_pdl(hl_compact_kernel, dim3(compact_ctas(ngroups)),
                         dim3(HL_COMPACT_THREADS), 0, s, false, *a);
}

/* Bounding box of an interleaved (x, y) list: bbox = {xmin, ymin, xmax, ymax}
 * (the reference's _findMinMaxCoordinates, okano_3_0/HoughLine.cu:287-334,
 * done on the device).  Every CTA writes its own box; the last one to finish
 * combines them and writes the result straight into mapped host memory, which
 * the host reads after its one synchronisation. */
#define BBOX_THREADS 512
__device__ __forceinline__ int4 bbox_join(int4 a, int4 b)
{
    return make_int4(min(a.x, b.x), min(a.y, b.y), max(a.z, b.z), max(a.w, b.w));
}
__device__ __forceinline__ int4 bbox_block(int4 b, int4 *s)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        b = bbox_join(b, make_int4(__shfl_xor_sync(FULL, b.x, o), __shfl_xor_sync(FULL, b.y, o),
                                   __shfl_xor_sync(FULL, b.z, o), __shfl_xor_sync(FULL, b.w, o)));
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
        s[threadIdx.x >> 5] = b;
    __syncthreads();
    for (int w = 0; w < BBOX_THREADS / 32; w++)
        b = bbox_join(b, s[w]);
    return b;
}
__global__ void __launch_bounds__(BBOX_THREADS)
hl_bbox_kernel(const int *xy, int n, int4 *part, unsigned *ticket, int *bbox)
{
    __shared__ int4 s[BBOX_THREADS / 32];
    __shared__ bool s_last;
    const int4 none = make_int4(0x7fffffff, 0x7fffffff, (int)0x80000000, (int)0x80000000);
    int4 b = none;
    for (int i = blockIdx.x * BBOX_THREADS + threadIdx.x; i < n; i += gridDim.x * BBOX_THREADS) {
        const int2 p = reinterpret_cast<const int2 *>(xy)[i];
        b = bbox_join(b, make_int4(p.x, p.y, p.x, p.y));
    }
    b = bbox_block(b, s);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = b;
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last)
        return;
    __threadfence();
    b = threadIdx.x < gridDim.x ? __ldcg(part + threadIdx.x) : none;
    b = bbox_block(b, s);
    if (threadIdx.x == 0) {
        *reinterpret_cast<int4 *>(bbox) = b;
        *ticket = 0u;
        __threadfence_system();
    }
}

cudaError_t hl_launch_bbox(const int *xy, int n, int4 *part, unsigned *ticket, int *bbox,
                           cudaStream_t s)
{
    const int blocks =
        std::max(1, std::min((n + 4 * BBOX_THREADS - 1) / (4 * BBOX_THREADS), HL_BBOX_CTAS));
    hl_bbox_kernel<<<blocks, BBOX_THREADS, 0, s>>>(xy, n, part, ticket, bbox);
    return cudaGetLastError();
}
