/*
 * hl_vote.cu -- stage (b): (theta, rho) int32 voting.
 *
 * Vote rule (okano_3_0/HoughLine.cu:86-130): an edge point (x, y) adds one
 * to bin (k, trunc(fl(x*cos_k) + fl(y*sin_k))) for every k.  The products and
 * the sum are rounded separately (packed f32x2 products as fma(a, b, +0) and
 * a packed add: no FMA contraction, see f2_mul), the float is truncated
 * toward zero (the reference's +-0.5 step after the (int) cast is a no-op),
 * and cos_k/sin_k come from the GPU-evaluated table.
 *
 * Work decomposition.  A work item is one theta slice (32 thetas) of one
 * region of the image, a rectangle of compaction tiles.  Its counts live in
 * shared memory as acc[row][column], where each column's rows start at the
 * lowest rho the rectangle reaches at that theta: over the slice the windows
 * follow the rectangle's sinusoid, so about its diagonal's number of rows holds
 * every vote of its points.  No vote falls outside and none is executed twice
 * -- fixed rho windows over all points executed 1.4 to 1.6 votes a useful one,
 * a tile being voted by every window its rho range over the slice meets.
 * A warp votes 8 points at a time on the diagonal schedule (DiagTab): at every
 * step its 32 lanes add to 32 different theta columns -- 32 different banks --
 * so every shared-memory reduction is conflict-free and no two lanes ever hit
 * one address.
 *
 * Pipeline.  Persistent CTAs of one producer warp and consumer warps that
 * meet only on mbarriers.  The producer takes items heaviest-first from a
 * global counter.  For an item it evaluates the vote rule at the rectangle's
 * corners (every rounded step is monotone in x and in y, so they bound every
 * point's rho exactly), reads the point offsets of the rectangle's tile rows
 * -- contiguous ranges of the tile-major point list, 16-byte aligned because
 * the compaction pads every tile to an even number of float2 entries -- and
 * publishes it as a segment (double-buffered descriptor).  The runs, laid end
 * to end, form the item's point stream: it is copied in batches into a ring of
 * HL_VOTE_SLOTS shared-memory slots with cp.async.bulk (completing on the slot's
 * full barrier); the consumer warps take blocks of 32 points of a slot in turn,
 * vote them straight from shared memory and arrive on the slot's empty barrier,
 * which the producer waits on before refilling it.  The producer moves on to
 * the next item as soon as the current one is issued.
 * Where regions would get small (rho steps below 1) or a merge is not worth its
 * launch, a block is voted in windows instead: an item takes the tiles that may
 * reach its rows (hl_band.h), tests every vote's row against them, and its rows are
 * final; a window heavier than a CTA's share is voted in parts of its points.
 * When an item is voted the consumers read it and clear what they read.  The
 * only item of its block is final: when peaks are wanted, its bins above the
 * threshold go to the accumulator, which is zero otherwise (the peak rule needs
 * no others, and the tail clears them again), and onto the candidate list --
 * writing whole accumulators cost a batch of 256 images 670 MB and a fifth of
 * its vote kernel; when the accumulator itself is wanted, all of it.  Other
 * items go to a scratch slab that hl_merge_kernel sums.
 * A whole image that one CTA votes alone (batches) but whose range exceeds the
 * window is voted in segments of a sliding window: tiles are taken in bands
 * across the slice's middle normal, the rows that no later band reaches are
 * stored, and the rest moves down.
 *
 * Per vote: half a packed multiply of x and of y each for two thetas, half a
 * packed add and half a packed magic-constant add (the float -> integer, see
 * RHO_MAGIC), one shift-and-add (the column's address, window base and the
 * constant's bits are one register) and one red.shared, plus an eighth of a
 * point load; no clamp and no branch per vote.
 *
 * Bound by instruction issue: 5 instructions a warp-vote in the loop, 1.6 of an
 * SM's cycles against the 1.13 of the shared-memory atomics alone, and the
 * items' edges (first copies, store, barriers) about a quarter of the time.
 * 4096 x 4096, T = 720: 92 us (fixed rho windows 118 us), with the slab merge 109
 * (128).  256 images of 256..2048 a side, T = 360: 854 us (1267).  2048 points a
 * slot: 1024 make every warp wait on a barrier for every block it votes (4096 x 4096
 * 158 against 153 us, the batch 1364 against 1318).
 *
 * Bounds: every voted point lies in the item's rectangle (or band), whose rows
 * the window holds; the list's sentinel (+infinity pads an odd tile) and stale
 * ring data vote 0 at the place of a real point; a window's votes are clamped to it
 * one by one.  A launch whose compaction reported an error votes nothing.
 * After the start there is no block-wide barrier, and every mbarrier wait is
 * bounded: a time-out sets a status bit that the host reads with the result
 * and an abort flag on which every other waiting warp gives up too; the
 * producer then waits (bounded) for its copies in flight before exiting.
 */
#include "hl_internal.h"
#include "hl_band.h"
#include "hl_device.cuh"

#include <algorithm>

#define FULL 0xffffffffu
#define MBAR_WAIT_LIMIT (1 << 14)
/* float2 entries of one ring slot (runs are gap-free: the compaction pads
 * every tile to an even number of points, 16 bytes) */
#define SLOT_CAP HL_VOTE_CHUNK

/* ---- mbarrier + bulk copy ---------------------------------------------- */
__device__ __forceinline__ unsigned smem_u32(const void *p)
{
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned n)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(n)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar,
                                               unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                     smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src,
                                         unsigned bytes,
                                         unsigned long long *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
/* bounded wait for the phase with the given parity (false on time-out);
 * each try_wait may suspend the warp for up to about a microsecond instead
 * of spinning, leaving issue slots to working warps */
__device__ __forceinline__ bool mbar_wait_sleep(unsigned long long *bar,
                                                unsigned parity)
{
    const unsigned a = smem_u32(bar);
    for (int i = 0; i < MBAR_WAIT_LIMIT; i++) {
        unsigned ok;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], "
            "%2, %3; selp.u32 %0, 1, 0, p; }"
            : "=r"(ok)
            : "r"(a), "r"(parity), "r"(1000u)
            : "memory");
        if (ok)
            return true;
    }
    return false;
}

/* An item as the producer hands it to the consumers, or the end of the work
 * (item < 0). */
struct VoteSeg {
    int32_t *acc;                      /* the image's accumulator */
    int item;                          /* its index, or -1 */
    int img, k0;                       /* image, first theta of the slice */
    int mode;                          /* CV_* (CV_EXACT: every row tested) */
    int total;                         /* points of its stream */
    int rho_min, R, thr;               /* the image's */
    int slab;                          /* see hl_vote_item */
    int win;                           /* an item of one window: see hl_vote_item */
    int last, adv;                     /* the item's last segment; rows to slide */
    int rows;                          /* rows its votes can reach; of a window */
    float margin;                      /* one rho bin in pixels */
    float c[HL_SLICE], s[HL_SLICE];    /* cos / sin of the slice's thetas */
    int base[HL_SLICE];                /* rho of each column's row 0 */
    int gb[4], gn[4], go[4];           /* the slab's column groups */
};

/* The lane's tables of an item: cos / sin of its columns as f2x pairs of
 * consecutive steps (DiagTab's order), and key[i] with 128 * bits + key[i] the
 * shared address of the vote at step i (bits: the magic-constant sum). */
struct VoteTab {
    f2x c[4], s[4];
    unsigned key[8];
};

/* the vote at relative shared address rel if it lies below lim, else at the same
 * column of the row there: a predicated reduction costs branches (16 images of 1000 x
 * 900, step 0.1: 193 us a call, 174 so) */
__device__ __forceinline__ void red_below(unsigned rel, unsigned lim, unsigned acc_base)
{
    red_smem(acc_base + min(rel, lim | (rel & 127u)));
}

/* 32 points from pts on, 8 a round, 8 votes of each a lane.  WIN: the table's keys
 * are relative to the window, and votes past lim, its bytes, go to the row after. */
template <bool UNIT, int CV, bool WIN>
__device__ __forceinline__ void vote_rounds(const float2 *pts, const VoteTab &t, f2x ir,
                                            unsigned lim, unsigned acc_base)
{
    pts += threadIdx.x & 7;
#pragma unroll
    for (int r = 0; r < 32; r += 8) {
        const float2 q = pts[r];
        const f2x X = f2_pack(q.x, q.x), Y = f2_pack(q.y, q.y);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            unsigned r0, r1;
            diag_bits<UNIT, CV>(X, Y, t.c[i], t.s[i], ir, r0, r1);
            if (WIN) {
                red_below(128u * r0 + t.key[2 * i], lim, acc_base);
                red_below(128u * r1 + t.key[2 * i + 1], lim, acc_base);
            } else {
                red_smem(128u * r0 + t.key[2 * i]);
                red_smem(128u * r1 + t.key[2 * i + 1]);
            }
        }
    }
}

/* Points whose |rho| may reach 2^22 (or that a window promised to hold and does
 * not): point by point, a lane a theta, by the conversion instruction, every
 * row tested. */
template <bool UNIT>
__device__ __noinline__ void vote_clipped(const float2 *pts, unsigned real, const VoteSeg &g,
                                          int rows, int *acc, float irho)
{
    const int lane = threadIdx.x & 31;
    const float c = g.c[lane], s = g.s[lane];
    const int base = g.base[lane];
    for (; real; real &= real - 1) {
        const float2 q = pts[__ffs(real) - 1];
        const int row = rho_of<UNIT>(q.x, q.y, c, s, irho) - base;
        if ((unsigned)row < (unsigned)rows)
            atomicAdd(acc + row * HL_SLICE + lane, 1);
    }
}

/* Floor, ceil or truncation by sign for a warp's points: which blocks lie on one
 * side of rho 0 over the whole slice (a sinusoid has at most one zero in it, so its
 * ends tell, with a bin to spare) is looked at once. */
template <bool UNIT, bool WIN>
__device__ __forceinline__ void vote_cv(const float2 *pts, float2 q, bool there, int mode,
                                        const VoteTab &t, f2x ir, const VoteSeg &g, unsigned lim,
                                        unsigned acc_base)
{
    int cv = mode;
    if (mode == CV_SIGN) {
        const float v0 = q.x * g.c[0] + q.y * g.s[0];
        const float v1 = q.x * g.c[HL_SLICE - 1] + q.y * g.s[HL_SLICE - 1];
        if (__all_sync(FULL, !there || fminf(v0, v1) > g.margin))
            cv = CV_FLOOR;
        else if (__all_sync(FULL, !there || fmaxf(v0, v1) < -g.margin))
            cv = CV_CEIL;
    }
    if (cv == CV_FLOOR)
        vote_rounds<UNIT, CV_FLOOR, WIN>(pts, t, ir, lim, acc_base);
    else if (cv == CV_CEIL)
        vote_rounds<UNIT, CV_CEIL, WIN>(pts, t, ir, lim, acc_base);
    else
        vote_rounds<UNIT, CV_SIGN, WIN>(pts, t, ir, lim, acc_base);
}

/* A warp's block of a slot: 32 places, n of them filled.  They are looked at
 * once, a lane a place: the ones with no point (past the end, or the list's
 * sentinel) are filled with one of the block's points, whose surplus votes the
 * warp takes off again, so that no vote needs a test -- in a window item, where
 * every vote is tested, with the sentinel.  Conflict-free red.shared alone take
 * 1.13 cycles a warp-vote an SM; the floor 1.5, truncation by sign 2.15
 * (micro-benchmark, 31 warps). */
template <bool UNIT, bool WIN>
__device__ __forceinline__ void vote_block(float2 *pts, int n, int mode, const VoteTab &t,
                                           f2x ir, const VoteSeg &g, int *acc, unsigned acc_base,
                                           float irho)
{
    const int lane = threadIdx.x & 31;
    const bool win = WIN && g.win;
    const float2 q = pts[lane];
    const bool there = lane < n && q.x < 1.0e29f;
    const unsigned real = __ballot_sync(FULL, there);
    if (!real)
        return;
    if (mode == CV_EXACT) {
        vote_clipped<UNIT>(pts, real, g, g.rows, acc, irho);
        return;
    }
    if (real != FULL) {
        const float2 f = win ? make_float2(__int_as_float(0x7f800000), 0.0f)
                               : pts[__ffs(real) - 1];
        if (!there) {
            pts[lane] = f;
            /* the slot is refilled by the async proxy */
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        if (!win) {
            const int row = rho_of<UNIT>(f.x, f.y, g.c[lane], g.s[lane], irho) - g.base[lane];
            atomicSub(acc + row * HL_SLICE + lane, 32 - __popc(real));
        }
        __syncwarp();
    }
    if (win)
        vote_cv<UNIT, true>(pts, q, there, mode, t, ir, g, 128u * (unsigned)g.rows, acc_base);
    else
        vote_cv<UNIT, false>(pts, q, there, mode, t, ir, g, 0u, acc_base);
}

/* Bounded wait that also gives up as soon as another warp of the CTA has
 * given up (*abort_flag set).  A time-out sets the flag and the status bit;
 * false means: leave the kernel. */
__device__ __forceinline__ bool mbar_wait_ab(unsigned long long *bar,
                                             unsigned parity, int *abort_flag,
                                             int *status)
{
    const unsigned a = smem_u32(bar);
    for (int i = 0; i < MBAR_WAIT_LIMIT; i++) {
        unsigned ok;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], "
            "%2, %3; selp.u32 %0, 1, 0, p; }"
            : "=r"(ok)
            : "r"(a), "r"(parity), "r"(1000u)
            : "memory");
        if (ok)
            return true;
        if (*(volatile int *)abort_flag)
            return false;
    }
    if ((threadIdx.x & 31) == 0)
        atomicOr(status, HL_ST_VOTE_TIMEOUT);
    *(volatile int *)abort_flag = 1;
    return false;
}

struct VoteSmem {
    unsigned long long full[HL_VOTE_SLOTS];
    unsigned long long empty[HL_VOTE_SLOTS];
    unsigned long long seg_full[2];    /* producer -> consumers */
    unsigned long long seg_empty[2];   /* consumers -> producer */
    unsigned long long cbar;           /* barrier of the consumer warps */
    int abort;                         /* a warp gave up waiting */
    VoteSeg seg[2];
    int run_s[HL_VOTE_RUNS];           /* producer: the runs' first points */
    int rpre[HL_VOTE_RUNS + 1];        /* their stream positions */
    alignas(16) float2 raw[HL_VOTE_SLOTS][SLOT_CAP];
};

#define VOTE_FIXED ((sizeof(VoteSmem) + 127) / 128 * 128)

/* the window's rows and, for items of one window, the one that takes the votes past it */
size_t hl_vote_smem_bytes(int win_rows)
{
    return VOTE_FIXED + (size_t)(win_rows + 1) * HL_SLICE * sizeof(int);
}

int hl_vote_max_rows(void)
{
    const size_t cap = 227u * 1024u;
    return (int)((cap - VOTE_FIXED) / (HL_SLICE * sizeof(int)) - 1) & ~7;
}

/* barrier of the consumer warps (bounded wait): one arrival a warp, after its
 * lanes' accesses -- an arrival a thread serialises a thousand of them on one
 * shared-memory word */
__device__ __forceinline__ bool cons_sync(VoteSmem &sm, unsigned &par,
                                          int *status)
{
    __syncwarp();
    if ((threadIdx.x & 31) == 0)
        mbar_arrive(&sm.cbar);
    const bool ok = mbar_wait_ab(&sm.cbar, par, &sm.abort, status);
    par ^= 1u;
    return ok;
}

/* Producer warp: takes items, publishes each as a segment and streams its
 * points into the ring.  It runs ahead of the consumers by up to the ring's
 * depth, so the next item's setup and first copies overlap the current item's
 * last votes. */
template <bool WIN>
__device__ __forceinline__ void vote_producer(const hl_vote_args &a, VoteSmem &sm)
{
    const int lane = threadIdx.x & 31;
    unsigned seq = 0;    /* batches issued */
    unsigned nseg = 0;   /* segments published */
    bool ok = true;
    /* nothing is voted after a failed compaction: its offsets are not valid */
    const bool skip = *(volatile int *)a.status != 0;
    while (ok) {
        /* in order of arrival, the first item too: under programmatic launch
         * some CTAs start late */
        unsigned t = 0;
        if (lane == 0)
            t = atomicAdd(a.work, 1u) - a.work_base;
        t = __shfl_sync(FULL, t, 0);
        const bool have = t < (unsigned)a.nitems;
        hl_vote_item it = {};
        hl_vote_img im = a.img0;
        if (have) {
            it = a.items[t];
            if (a.imgs)
                im = a.imgs[it.img];
        }
        const bool win = WIN && it.win;
        const int tx0 = it.tx & 0xffff, txn = it.tx >> 16;
        const int ty0 = it.ty & 0xffff, tyn = it.ty >> 16;
        /* the columns past T vote like the last theta: their counts are
         * cleared with the others' and stored as zero */
        const int k = min(it.slice * HL_SLICE + lane, a.T - 1);
        const float cl = a.cosv[k], sl = a.sinv[k];
        /* rho range of each theta over the rectangle */
        float lo = 3.0e38f, hi = -3.0e38f;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float x = (float)((i & 1) ? min((tx0 + txn) * HL_TILE_W, im.w) - 1
                                            : tx0 * HL_TILE_W);
            const float y = (float)((i & 2) ? min((ty0 + tyn) * HL_TILE_H, im.h) - 1
                                            : ty0 * HL_TILE_H);
            const float v = rho_f<false>(x, y, cl, sl, a.irho);
            lo = fminf(lo, v);
            hi = fmaxf(hi, v);
        }
        const bool slide = it.nseg > 1 && !win;
        const float ctx = 0.5f * (float)(im.w - 1), cty = 0.5f * (float)(im.h - 1);
        int base = slide || win
                       ? __float2int_rd(rho_f<false>(ctx, cty, cl, sl, a.irho)) + it.off0
                       : __float2int_rz(lo);
        int top = __float2int_rz(hi);
        bool clip = false;
        if (have && !slide && !win && __any_sync(FULL, top - base >= a.win_rows)) {
            if (lane == 0)   /* the plan promised more rows than there are */
                atomicOr(a.status, HL_ST_RHO_OUT_OF_RANGE);
            clip = true;
        }
        const int wrows = win ? min(it.adv, a.win_rows) : a.win_rows;
        if (!slide)
            top = min(top, base + wrows - 1);
        int mode = a.exact ? CV_EXACT
                           : (!__any_sync(FULL, lo < 0.0f)
                                  ? CV_FLOOR
                                  : (!__any_sync(FULL, hi > 0.0f) ? CV_CEIL : CV_SIGN));
        const bool mixed = mode == CV_SIGN;
        /* sliding: the middle theta's normal in rho units a tile */
        const int km = min(it.slice * HL_SLICE + HL_SLICE / 2, a.T - 1);
        const float sm_ = slide ? a.sinv[km] * a.irho : win ? a.sinv[km] : 0.0f;
        float cm = slide ? a.cosv[km] * a.irho : win ? a.cosv[km] : 0.0f;
        if (!win)
            cm = copysignf(fmaxf(fabsf(cm), 1.0e-9f), cm);
        const float icm = 1.0f / (cm * HL_TILE_W);
        const float x0 = __fmul_rn(ctx - HL_TILE_W / 2, 1.0f / HL_TILE_W);
        const bool wide = txn == im.tiles_x && !slide && !win;
        const int nsegs = have ? max(it.nseg, 1) : 1;

        for (int sj = 0; sj < nsegs && ok; sj++, base += slide ? it.adv : 0) {
        const int rows = __reduce_max_sync(FULL, max(min(top, base + wrows - 1) - base + 1, 0));
        if (clip)
            mode = CV_EXACT;   /* every row tested */
        if (win && mixed)   /* rho 0 truncates from both sides */
            mode = !__any_sync(FULL, base < 1)
                       ? CV_FLOOR
                       : (!__any_sync(FULL, base + rows > 0) ? CV_CEIL : CV_SIGN);
        if (slide && mixed)   /* by the segment's own rows */
            mode = !__any_sync(FULL, base < 0)
                       ? CV_FLOOR
                       : (!__any_sync(FULL, base + a.win_rows > 0) ? CV_CEIL : CV_SIGN);
        /* the runs, lane and every 32nd after it: one a tile row, or one for a
         * rectangle as wide as the image; a window's item two a tile row.  Few
         * runs are one round: a lane's are looked up one after the other */
        const int nruns = !have || skip ? 0
                          : wide        ? 1
                          : win      ? 2 * min(tyn - sj * (HL_VOTE_RUNS / 2), HL_VOTE_RUNS / 2)
                                        : min(tyn, HL_VOTE_RUNS);
        int st[HL_VOTE_RUNS / 32], en[HL_VOTE_RUNS / 32];
#pragma unroll
        for (int q = 0; q < HL_VOTE_RUNS / 32; q++) {
            st[q] = en[q] = 0;
            if (32 * q < nruns) {
                const int r = 32 * q + lane;
                int ta = 0, tb = txn;   /* the run's tiles, from tx0 */
                const int ty = ty0 + (win ? sj * (HL_VOTE_RUNS / 2) + r / 2 : r);
                const float y = (float)(ty * HL_TILE_H + HL_TILE_H / 2) - cty;
                if (win)
                    hl_band_window(r & 1, it.lo, it.hi, it.tang, cm, sm_, HL_TILE_W / 2 - ctx, y,
                                   txn, &ta, &tb);
                if (slide)
                    hl_band_tiles(sj, nsegs, it.adv, it.half, __fmul_rn(y, sm_), cm, icm, x0, txn,
                                  &ta, &tb);
                if (r < nruns && tb > ta) {
                    const int t0 = ty * im.tiles_x + tx0;
                    st[q] = im.tile_off[t0 + ta];
                    en[q] = im.tile_off[wide ? (ty0 + tyn) * im.tiles_x : t0 + tb];
                }
            }
        }
        __syncwarp();   /* the previous segment's runs are no longer read */
        /* laid end to end a lane's after the other's: the order is free */
        const int rounds = (nruns + 31) / 32, nslots = 32 * rounds;
        int sum = 0;
#pragma unroll
        for (int q = 0; q < HL_VOTE_RUNS / 32; q++)
            sum += en[q] - st[q];
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t1 = __shfl_up_sync(FULL, incl, o);
            if (lane >= o)
                incl += t1;
        }
        const int all = __shfl_sync(FULL, incl, 31);
        int pos = incl - sum;
#pragma unroll
        for (int q = 0; q < HL_VOTE_RUNS / 32; q++)
            if (q < rounds) {
                sm.run_s[rounds * lane + q] = st[q];
                sm.rpre[rounds * lane + q] = pos;
                pos += en[q] - st[q];
            }
        if (lane == 31)
            sm.rpre[nslots] = all;
        /* a part of them, from and to even places */
        const int np = WIN ? max(it.nparts, 1) : 1, part = WIN ? it.part : 0;
        const int from = (int)((long long)all * part / np) & ~1;
        const int to = part + 1 < np ? (int)((long long)all * (part + 1) / np) & ~1 : all;
        const int total = to - from;

        /* publish the segment once the consumers are done with the one that
         * last used its slot */
        const int ds = (int)(nseg & 1u);
        if (nseg >= 2 && !mbar_wait_ab(&sm.seg_empty[ds], ((nseg >> 1) - 1u) & 1u, &sm.abort,
                                       a.status)) {
            ok = false;
            break;
        }
        VoteSeg &g = sm.seg[ds];
        g.c[lane] = cl;
        g.s[lane] = sl;
        g.base[lane] = base;
        if (lane == 0) {
            g.acc = im.acc;
            g.item = have ? (int)t : -1;
            g.img = it.img;
            g.k0 = it.slice * HL_SLICE;
            g.mode = mode;
            g.margin = 1.0f / a.irho;
            g.total = total;
            g.rho_min = im.rho_min;
            g.R = im.R;
            g.thr = im.threshold;
            g.slab = it.slab;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                g.gb[q] = it.gb[q];
                g.gn[q] = it.gn[q];
                g.go[q] = it.go[q];
            }
            if (WIN)
                g.win = win;
            g.last = sj == nsegs - 1;
            g.adv = it.adv;
            g.rows = rows;
        }
        __syncwarp();
        if (lane == 0)
            mbar_arrive(&sm.seg_full[ds]);
        nseg++;

        /* batch b is stream range [from + b * SLOT_CAP, ...): lane i copies the part
         * of run r0 + i overlapping it; a ballot finds the first run of the
         * next batch */
        const int nb = (total + SLOT_CAP - 1) / SLOT_CAP;
        int r0 = 0;
        for (int b = 0; b < nb && ok; b++) {
            const int slot = (int)(seq % HL_VOTE_SLOTS);
            if (seq >= HL_VOTE_SLOTS &&
                !mbar_wait_ab(&sm.empty[slot], ((seq / HL_VOTE_SLOTS) - 1u) & 1u, &sm.abort,
                              a.status)) {
                ok = false;
                break;
            }
            const int s0 = from + b * SLOT_CAP;
            const int e0 = min(to, s0 + SLOT_CAP);
            if (lane == 0)
                mbar_expect_tx(&sm.full[slot], (unsigned)(e0 - s0) * 8u);
            __syncwarp();
            /* runs from r0 on: every run ending at or before e0 lies wholly in
             * this batch; the first one reaching past e0 is shared with the
             * next batch and ends the scan */
            int nextr = nslots;
            for (int rb = r0; rb < nslots; rb += 32) {
                const int r = rb + lane;
                bool past = false;
                if (r < nslots) {
                    const int rs = sm.rpre[r], re = sm.rpre[r + 1];
                    const int ps = max(s0, rs), pe = min(e0, re);
                    if (pe > ps)
                        bulk_g2s(&sm.raw[slot][ps - s0], im.pts + sm.run_s[r] + (ps - rs),
                                 (unsigned)(pe - ps) * 8u, &sm.full[slot]);
                    past = re > e0;
                }
                const unsigned pm = __ballot_sync(FULL, past);
                if (pm) {
                    nextr = rb + __ffs(pm) - 1;
                    break;
                }
            }
            r0 = nextr;
            seq++;
        }
        }
        if (!have)
            break;
    }
    if (!ok) {
        /* gave up: wait (bounded) for the copies still in flight before
         * the CTA may exit */
        for (unsigned b = seq - min(seq, (unsigned)HL_VOTE_SLOTS); b < seq; b++)
            mbar_wait_sleep(&sm.full[b % HL_VOTE_SLOTS], (b / HL_VOTE_SLOTS) & 1u);
    }
}

/* WIN: some of the items are of one window each.  Their selection and tests cost the
 * others registers: 256 uneven images 1042 us in the one form for both, 1021 apart. */
template <bool UNIT, bool WIN>
__global__ void __launch_bounds__(1024, 1)
hl_vote_kernel(hl_vote_args a)
{
    extern __shared__ __align__(128) unsigned char vote_raw[];
    VoteSmem &sm = *reinterpret_cast<VoteSmem *>(vote_raw);
    int *s_acc = reinterpret_cast<int *>(vote_raw + VOTE_FIXED);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nthr = blockDim.x, nwarps = nthr >> 5;
    const int ncons = nwarps - 1;               /* consumer warps 1..nwarps-1 */
    /* the window starts at zero (before the wait for the previous launch:
     * shared memory only); after each item the consumers clear what it used */
    {
        int4 *z = reinterpret_cast<int4 *>(s_acc);
        for (int i = tid; i < a.win_rows * (HL_SLICE / 4); i += nthr)
            z[i] = make_int4(0, 0, 0, 0);
    }
    hl_pdl_begin();
    if (tid == 0) {
        for (int i = 0; i < HL_VOTE_SLOTS; i++) {
            mbar_init(&sm.full[i], 1);
            mbar_init(&sm.empty[i], (unsigned)ncons);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&sm.seg_full[i], 1);
            mbar_init(&sm.seg_empty[i], (unsigned)ncons);
        }
        mbar_init(&sm.cbar, (unsigned)ncons);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        sm.abort = 0;
    }
    /* the only block-wide barrier: from here on the producer and the
     * consumers meet on mbarriers, every wait bounded */
    __syncthreads();
    if (warp == 0) {
        vote_producer<WIN>(a, sm);
        return;
    }

    const int cw = warp - 1;
    const unsigned acc_base = smem_u32(s_acc);
    const f2x ir = f2_pack(a.irho, a.irho);
    unsigned seq = 0, nseg = 0, cpar = 0;
    bool full = false;   /* the candidate list */
    while (true) {
        const int ds = (int)(nseg & 1u);
        if (!mbar_wait_ab(&sm.seg_full[ds], (nseg >> 1) & 1u, &sm.abort, a.status))
            return;
        nseg++;
        const VoteSeg &g = sm.seg[ds];
        if (g.item < 0)
            return;
        const int total = g.total, mode = g.mode;
        {
            VoteTab tab;
            {
                const int p = lane & 7, j = lane >> 3;
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    const int c0 = 8 * j + ((p + i) & 7), c1 = 8 * j + ((p + i + 1) & 7);
                    tab.c[i / 2] = f2_pack(g.c[c0], g.c[c1]);
                    tab.s[i / 2] = f2_pack(g.s[c0], g.s[c1]);
                    const unsigned at = WIN && g.win ? 0u : acc_base;
                    tab.key[i] = at + 4u * (unsigned)c0 -
                                 128u * (unsigned)(RHO_MAGIC_BITS + g.base[c0]);
                    tab.key[i + 1] = at + 4u * (unsigned)c1 -
                                     128u * (unsigned)(RHO_MAGIC_BITS + g.base[c1]);
                }
            }
            /* vote the item's blocks in turn, freeing each slot */
            int i = 32 * cw;   /* the warp's next point of the slot */
            for (int b = 0; b * SLOT_CAP < total; b++) {
                const int slot = (int)(seq % HL_VOTE_SLOTS);
                if (!mbar_wait_ab(&sm.full[slot], (seq / HL_VOTE_SLOTS) & 1u, &sm.abort,
                                  a.status))
                    return;
                seq++;
                const int n = min(SLOT_CAP, total - b * SLOT_CAP);
                for (; i < n; i += 32 * ncons)
                    vote_block<UNIT, WIN>(sm.raw[slot] + i, n - i, mode, tab, ir, g, s_acc,
                                          acc_base, a.irho);
                i -= n;
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(&sm.empty[slot]);
            }
        }

        if (WIN && g.win && !g.last) {   /* more rows of tiles for the same window */
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&sm.seg_empty[ds]);
            continue;
        }
        /* the item is voted: store it and clear what is read, lane = column */
        if (!cons_sync(sm, cpar, a.status))
            return;
        const int k = g.k0 + lane;
        const bool kvalid = k < a.T;
        const int rb = g.base[lane] - g.rho_min;   /* the accumulator row of row 0 */
        int *col = s_acc + lane;
        if (WIN && g.win && cw == 0)   /* the votes past the window */
            col[g.rows * HL_SLICE] = 0;
        if (g.slab < 0) {
            /* the rows that are final: all of them, or those below the next
             * segment's window */
            const bool last = g.last;
            const int nr = last ? g.rows : g.adv;
            if (a.add) {   /* several items of a block, no slabs */
                for (int i = cw; i < nr; i += ncons) {
                    const int v = col[i * HL_SLICE];
                    if (v) {
                        col[i * HL_SLICE] = 0;
                        if (kvalid && (unsigned)(i + rb) < (unsigned)g.R)
                            atomicAdd(g.acc + (size_t)(i + rb) * a.Tp + k, v);
                    }
                }
            } else if (a.cand.e) {
                /* only bins above the threshold matter (the peak rule compares
                 * them with each other): they go to the accumulator, which is
                 * zero otherwise, and onto the candidate list.  Four columns
                 * of a row a lane, as the window lies in shared memory. */
                const int thr = max(g.thr, 0), n4 = nr * (HL_SLICE / 4);
                int4 *w = reinterpret_cast<int4 *>(s_acc);
                for (int i0 = 32 * cw; i0 < n4; i0 += 32 * ncons) {
                    const int i = i0 + lane, c = 4 * (i & 7);
                    unsigned bits = 0;
                    int4 v = make_int4(0, 0, 0, 0);
                    if (i < n4) {
                        v = w[i];
                        w[i] = make_int4(0, 0, 0, 0);
                    }
                    const auto row = [&](int e) { return (i >> 3) + g.base[c + e] - g.rho_min; };
                    if (max(max(v.x, v.y), max(v.z, v.w)) > thr) {
                        const int x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            if (x[e] > thr && g.k0 + c + e < a.T &&
                                (unsigned)row(e) < (unsigned)g.R) {
                                g.acc[(size_t)row(e) * a.Tp + g.k0 + c + e] = x[e];
                                bits |= 1u << e;
                            }
                    }
                    note_warp(a.cand, g.img, bits, full, [&](int e) {
                        return (unsigned)row(e) * (unsigned)a.T + (unsigned)(g.k0 + c + e);
                    });
                }
            } else {
                /* the whole accumulator is asked for: row by row, the shear
                 * undone by each lane's own offset.  Rows that no vote reaches
                 * stay as they are, zero. */
                const int lo = __reduce_min_sync(FULL, rb);
                const int hi = __reduce_max_sync(FULL, rb) + nr;
                for (int r = max(lo, 0) + cw; r < min(hi, g.R); r += ncons) {
                    const unsigned i = (unsigned)(r - rb);
                    if (i < (unsigned)nr) {
                        g.acc[(size_t)r * a.Tp + k] = kvalid ? col[i * HL_SLICE] : 0;
                        col[i * HL_SLICE] = 0;
                    }
                }
            }
            if (!last) {
                /* rows [adv, win_rows) move to the window's start (the plan
                 * keeps adv at least half the window) */
                if (!cons_sync(sm, cpar, a.status))
                    return;
                int4 *w = reinterpret_cast<int4 *>(s_acc), *f = w + nr * (HL_SLICE / 4);
                for (int i = 32 * cw + lane; i < (a.win_rows - nr) * (HL_SLICE / 4);
                     i += 32 * ncons) {
                    w[i] = f[i];
                    f[i] = make_int4(0, 0, 0, 0);
                }
            }
        } else {
            const int grp = lane >> 3, cc = lane & 7;
            const int gb = g.gb[grp], gn = g.gn[grp];
            const int most = max(max(g.gn[0], g.gn[1]), max(g.gn[2], g.gn[3]));
            const size_t at = ((size_t)g.slab + g.go[grp]) * 8 + cc;
            const int rows = g.rows;   /* that votes can reach */
            for (int q = cw; q < most; q += ncons) {
                int v[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    /* not the row of a window's other votes: it is cleared meanwhile */
                    const unsigned i = (unsigned)(4 * (gb + q) + u - rb);
                    v[u] = 0;
                    if (q < gn && i < (unsigned)rows) {
                        v[u] = col[i * HL_SLICE];
                        col[i * HL_SLICE] = 0;
                    }
                }
                if (q < gn) {
                    if (a.part16)
                        reinterpret_cast<uint2 *>(a.scratch)[at + (size_t)q * 8] =
                            make_uint2((unsigned)v[0] | ((unsigned)v[1] << 16),
                                       (unsigned)v[2] | ((unsigned)v[3] << 16));
                    else
                        reinterpret_cast<int4 *>(a.scratch)[at + (size_t)q * 8] =
                            make_int4(v[0], v[1], v[2], v[3]);
                }
            }
        }
        if (!cons_sync(sm, cpar, a.status))
            return;
        if (lane == 0)
            mbar_arrive(&sm.seg_empty[ds]);
    }
}

/* Blocks voted in several items: accumulator columns = sum of their slabs.  As
 * in hl_vote_kernel the bins above the image's threshold are stored and noted
 * as peak candidates, or every bin is stored (padding columns, thetas >= T,
 * zero).  A thread takes four rows of two columns: one
 * 16-byte load of every slab whose rows overlap (two with 32-bit counts), from
 * L2 where the vote launch just wrote them, eight in flight.  Bound by latency:
 * a block's slab list, then the slabs; where the slabs lie is the plan's, so no
 * header is read between.  4096 x 4096, T = 720: 18 us (23 us with headers that
 * the vote wrote, and CTAs for rows that no slab holds); 1913 x 1077, T = 360:
 * 8 us (13 us). */
#define MERGE_HDRS 64
template <bool P16>
__global__ void __launch_bounds__(256)
hl_merge_kernel(hl_merge_args a)
{
    __shared__ int4 s_b[MERGE_HDRS], s_n[MERGE_HDRS], s_o[MERGE_HDRS];   /* o: in scratch */
    __shared__ int s_hits;
    const int tid = threadIdx.x;
    hl_pdl_begin();
    const unsigned bi = blockIdx.x / a.chunks, chunk = blockIdx.x - bi * a.chunks;
    const hl_merge_block blk = a.blocks[bi];
    const int c0 = blk.lo + (int)chunk * 16;       /* the CTA's first row group */
    if (c0 >= blk.hi)
        return;
    const hl_vote_img &im = a.imgs ? a.imgs[blk.img] : a.img0;
    const int R = im.R;
    const int rg = c0 + (tid >> 4);                /* the thread's */
    const int g = (tid >> 2) & 3, cp = tid & 3;
    int v[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
    int hits = 0;
    for (int j0 = 0; j0 < blk.n; j0 += MERGE_HDRS) {
        /* the slabs that reach the CTA's rows */
        if (j0)
            __syncthreads();
        if (tid == 0)
            s_hits = 0;
        __syncthreads();
        if (tid < MERGE_HDRS && j0 + tid < blk.n) {
            const int4 *sl = reinterpret_cast<const int4 *>(a.slabs + blk.first + j0 + tid);
            const int4 h = sl[0], b = sl[1], n = sl[2], o = sl[3];
            if (h.y < c0 + 16 && h.z > c0) {
                const int at = atomicAdd(&s_hits, 1);
                s_b[at] = b;
                s_n[at] = n;
                s_o[at] = make_int4(h.x + o.x, h.x + o.y, h.x + o.z, h.x + o.w);
            }
        }
        __syncthreads();
        const int nj = s_hits;
        hits |= nj;
        /* the slabs' loads eight at a time (four with 32-bit counts) */
        constexpr int U = P16 ? 8 : 4;
        for (int j = 0; j < nj; j += U) {
            uint4 q[8];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int jj = min(j + u, nj - 1);
                const int rel = rg - reinterpret_cast<const int *>(&s_b[jj])[g];
                const bool ok = j + u < nj &&
                                (unsigned)rel < (unsigned)reinterpret_cast<const int *>(&s_n[jj])[g];
                const size_t at = ((size_t)reinterpret_cast<const int *>(&s_o[jj])[g] + rel) * 8 +
                                  2 * cp;
                if (P16) {
                    q[u] = ok ? __ldcg(reinterpret_cast<const uint4 *>(
                                    reinterpret_cast<const uint2 *>(a.scratch) + at))
                              : make_uint4(0u, 0u, 0u, 0u);
                } else {
                    const uint4 *p = reinterpret_cast<const uint4 *>(a.scratch) + at;
                    q[2 * u] = ok ? __ldcg(p) : make_uint4(0u, 0u, 0u, 0u);
                    q[2 * u + 1] = ok ? __ldcg(p + 1) : make_uint4(0u, 0u, 0u, 0u);
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (P16) {
                    v[0][0] += q[u].x & 0xffffu;
                    v[0][1] += q[u].x >> 16;
                    v[0][2] += q[u].y & 0xffffu;
                    v[0][3] += q[u].y >> 16;
                    v[1][0] += q[u].z & 0xffffu;
                    v[1][1] += q[u].z >> 16;
                    v[1][2] += q[u].w & 0xffffu;
                    v[1][3] += q[u].w >> 16;
                } else {
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        v[e][0] += (int)q[2 * u + e].x;
                        v[e][1] += (int)q[2 * u + e].y;
                        v[e][2] += (int)q[2 * u + e].z;
                        v[e][3] += (int)q[2 * u + e].w;
                    }
                }
            }
        }
    }
    /* rows that no slab reaches stay zero (see hl_vote_kernel) */
    if (!hits)
        return;
    const int k = blk.slice * HL_SLICE + 8 * g + 2 * cp;
    const bool k0v = k < a.T, k1v = k + 1 < a.T;
    int32_t *dst = im.acc + k;
    if (!a.cand.e) {   /* the whole accumulator is asked for */
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (4 * rg + u < R)
                *reinterpret_cast<int2 *>(dst + (size_t)(4 * rg + u) * a.Tp) =
                    make_int2(k0v ? v[0][u] : 0, k1v ? v[1][u] : 0);
        return;
    }
    const int thr = max(im.threshold, 0);
    unsigned bits = 0;   /* bit 2 u + e */
#pragma unroll
    for (int u = 0; u < 4; u++)
        if (max(v[0][u], v[1][u]) > thr && 4 * rg + u < R)
#pragma unroll
            for (int e = 0; e < 2; e++)
                if (v[e][u] > thr && (e ? k1v : k0v)) {
                    dst[(size_t)(4 * rg + u) * a.Tp + e] = v[e][u];
                    bits |= 1u << (2 * u + e);
                }
    /* every warp comes here once: without a look first, the counter of a full list
     * would grow with the accumulators */
    bool full = __any_sync(FULL, bits != 0) && *(volatile int *)a.cand.count > a.cand.cap;
    note_warp(a.cand, blk.img, bits, full, [&](int b) {
        return (unsigned)(4 * rg + (b >> 1)) * (unsigned)a.T + (unsigned)(k + (b & 1));
    });
}

cudaError_t hl_launch_merge(const hl_merge_args *a, cudaStream_t s)
{
    if (a->nblocks <= 0)
        return cudaSuccess;
    const unsigned long long grid = (unsigned long long)a->chunks * (unsigned)a->nblocks;
    if (grid > 0x7fffffffull)
        return cudaErrorInvalidConfiguration;
    return hl_launch_pdl(a->part16 ? hl_merge_kernel<true> : hl_merge_kernel<false>,
                         dim3((unsigned)grid), dim3(256), 0, s, false, *a);
}

cudaError_t hl_launch_vote(const hl_vote_args *a, int threads, int grid,
                           cudaStream_t s)
{
    const size_t smem = hl_vote_smem_bytes(a->win_rows);
    const bool unit = a->irho == 1.0f;
    const auto kernel = a->win ? (unit ? hl_vote_kernel<true, true> : hl_vote_kernel<false, true>)
                               : (unit ? hl_vote_kernel<true, false> : hl_vote_kernel<false, false>);
    const cudaError_t e = cudaFuncSetAttribute(
        kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess)
        return e;
    return hl_launch_pdl(kernel, dim3(grid), dim3(threads), smem, s, false, *a);
}

/* ---- voting over a coordinate list ------------------------------------------
 * The guidingset path (okano_3_0/HoughLine.cu:133-165): interleaved int (x, y),
 * any order, so no tile filter.  A CTA takes one theta slice (blockIdx.x), one
 * rho window of it (blockIdx.y) and one part of the points (blockIdx.z): the
 * parts spread a list over the chip however few slices there are.  A slice's
 * windows start at the lowest row its bounding box can reach and there are as
 * many as its range needs (one up to about 1200 x 1200), so most points vote
 * once a theta.  Votes go to shared memory on the vote kernel's diagonal
 * schedule, four rounds' points in flight; then the window's nonzero bins are
 * added to the accumulator (cleared before), a row of 32 thetas a reduction.
 * Bound by latency: clearing, voting and adding one window a CTA.  24 K points
 * of 1024 x 1024, T = 180, ncu: 10.7 us (100 us with every point broadcast to
 * every window of 66 CTAs); the whole call 147 -> 53 us. */
#define PTS_THREADS 1024
#define PTS_PART_MIN 1024      /* points a part at least holds */

static int points_max_rows(void)
{
    return (int)((227u * 1024u - 1024u) / (HL_SLICE * sizeof(int))) - 1;
}

template <bool UNIT, int CV>
__device__ __forceinline__ void points_vote(const int2 *xy, int p0, int p1, const DiagTab &t,
                                            f2x ir, int base, unsigned lim)
{
    const int warp = threadIdx.x >> 5, p = threadIdx.x & 7;
    constexpr int STEP = PTS_THREADS / 32 * 8;
    for (int g0 = p0 + warp * 8; g0 < p1; g0 += 4 * STEP) {
        float2 q[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int i = g0 + u * STEP + p;
            const int2 v = i < p1 ? xy[i] : make_int2(0, 0);
            q[u] = i < p1 ? make_float2((float)v.x, (float)v.y) : make_float2(1e30f, 0.0f);
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (g0 + u * STEP < p1)
                diag_point<UNIT, CV>(q[u].x, q[u].y, t, ir, base, lim);
    }
}

template <bool UNIT>
__global__ void __launch_bounds__(PTS_THREADS, 1)
hl_vote_points_kernel(hl_points_args a)
{
    extern __shared__ __align__(16) int s_pacc[];
    __shared__ float s_c[HL_SLICE], s_s[HL_SLICE];
    __shared__ int s_lo, s_hi;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int k0 = blockIdx.x * HL_SLICE;
    hl_pdl_begin();
    if (tid < HL_SLICE) {
        /* rho range of the slice over the bounding box: every rounded step
         * of the vote rule is monotone in x and in y, so the corners' values
         * bound it exactly */
        const float c = a.cosv[k0 + lane], s = a.sinv[k0 + lane];
        s_c[lane] = c;
        s_s[lane] = s;
        float lo = 3.0e38f, hi = -3.0e38f;
        if (k0 + lane < a.T)
            for (int i = 0; i < 4; i++) {
                const float v = rho_f<UNIT>((float)((i & 1) ? a.x1 : a.x0),
                                            (float)((i & 2) ? a.y1 : a.y0), c, s, a.irho);
                lo = fminf(lo, v);
                hi = fmaxf(hi, v);
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(FULL, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(FULL, hi, o));
        }
        if (lane == 0) {
            s_lo = max(__float2int_rd(lo) - a.rho_min, 0);
            s_hi = min(__float2int_ru(hi) - a.rho_min, a.R - 1);
        }
    }
    __syncthreads();
    const int w0 = s_lo + blockIdx.y * a.win_rows;   /* first row of the window */
    const int rows = min(a.win_rows, s_hi + 1 - w0);
    if (rows <= 0)
        return;
    int4 *z = reinterpret_cast<int4 *>(s_pacc);
    for (int i = tid; i < (rows + 1) * (HL_SLICE / 4); i += PTS_THREADS)
        z[i] = make_int4(0, 0, 0, 0);
    const int p0 = (int)((long long)a.n * blockIdx.z / gridDim.z);
    const int p1 = (int)((long long)a.n * (blockIdx.z + 1) / gridDim.z);
    DiagTab tab;
    diag_table(tab, s_c, s_s, smem_u32(s_pacc), lane);
    const f2x ir = f2_pack(a.irho, a.irho);
    const int row_base = a.rho_min + w0;
    __syncthreads();
    if (a.exact)   /* coordinates beyond the magic constant's range */
        points_vote<UNIT, CV_EXACT>(a.xy, p0, p1, tab, ir, row_base, (unsigned)rows);
    else if (row_base >= 1)
        points_vote<UNIT, CV_FLOOR>(a.xy, p0, p1, tab, ir, RHO_MAGIC_BITS + row_base,
                                    (unsigned)rows);
    else
        points_vote<UNIT, CV_SIGN>(a.xy, p0, p1, tab, ir, RHO_MAGIC_BITS + row_base,
                                   (unsigned)rows);
    __syncthreads();
    /* a warp a row, four rows in flight; the padding columns are left zero */
    const bool kvalid = k0 + lane < a.T;
    int *dst = a.acc + (size_t)w0 * a.Tp + k0 + lane;
    for (int r0 = warp * 4; r0 < rows; r0 += PTS_THREADS / 32 * 4) {
        int v[4];
#pragma unroll
        for (int u = 0; u < 4; u++)
            v[u] = r0 + u < rows && kvalid ? s_pacc[(r0 + u) * HL_SLICE + lane] : 0;
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (v[u])
                atomicAdd(dst + (size_t)(r0 + u) * a.Tp, v[u]);
    }
}

cudaError_t hl_launch_vote_points(hl_points_args *a, int sms, cudaStream_t s)
{
    const int slices = a->Tp / HL_SLICE;
    const int maxr = points_max_rows();
    const int nwin = std::max(1, (a->span + maxr - 1) / maxr);
    a->win_rows = std::max(1, std::min(maxr, (a->span + nwin - 1) / nwin));
    /* parts: one CTA an SM, all at once */
    const int parts = std::max(1, std::min(std::min((a->n + PTS_PART_MIN - 1) / PTS_PART_MIN,
                                                    sms / std::max(1, slices * nwin)), 64));
    const size_t smem = (size_t)(a->win_rows + 1) * HL_SLICE * sizeof(int);
    cudaError_t e = cudaMemsetAsync(a->acc, 0, sizeof(int) * (size_t)a->R * a->Tp, s);
    if (e != cudaSuccess)
        return e;
    const auto kernel = a->irho == 1.0f ? hl_vote_points_kernel<true> : hl_vote_points_kernel<false>;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess)
        return e;
    return hl_launch_pdl(kernel, dim3(slices, nwin, parts), dim3(PTS_THREADS), smem, s, false, *a);
}

/* Shared-memory atomic ceiling: every lane adds to its own bank, 8
 * independent addresses per thread per iteration, 1024 threads per CTA, two
 * CTAs per SM.  The counters are summed into *sink so nothing is dead. */
__global__ void __launch_bounds__(1024, 2)
hl_atomic_bench_kernel(int iters, int *sink)
{
    __shared__ int s[8 * 1024];
    const int tid = threadIdx.x;
    for (int i = tid; i < 8 * 1024; i += blockDim.x)
        s[i] = 0;
    __syncthreads();
    const int lane = tid & 31, warp = tid >> 5;
    int *base = s + (warp & 31) * 256 + lane;
    for (int it = 0; it < iters; it++) {
#pragma unroll
        for (int u = 0; u < 8; u++)
            atomicAdd(base + u * 32, 1);
    }
    __syncthreads();
    if (tid == 0) {
        int acc = 0;
        for (int i = 0; i < 8 * 1024; i += 97)
            acc += s[i];
        atomicAdd(sink, acc);
    }
}

cudaError_t hl_launch_atomic_bench(int iters, int *sink, cudaStream_t s,
                                   int *blocks_out, int *threads_out)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int blocks = sms * 2;
    hl_atomic_bench_kernel<<<blocks, 1024, 0, s>>>(iters, sink);
    if (blocks_out)
        *blocks_out = blocks;
    if (threads_out)
        *threads_out = 1024;
    return cudaGetLastError();
}
