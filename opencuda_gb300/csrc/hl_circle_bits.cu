/*
 * hl_circle_bits.cu -- HoughCircle's votes for radii up to HL_CIRCLE_DENSE_R,
 * counted without atomics.
 *
 * A cell's count is the number of edge pixels on the midpoint circle around it
 * (okano_3_0/HoughCircle.cu:187-245: the circle's offsets come in +- pairs, so
 * voting and gathering are the same sum; the points on the axes count twice).
 * The edge pixels are one bit each, and a thread counts 128 cells of a row at
 * once: for every offset it takes the 128 bits of the edge map at that offset
 * and adds them to nine bit planes with carry-save adders -- 2.5 three-input
 * logic operations a word an offset.  The local maxima (:321-370) are taken on
 * the bit planes too: v above the threshold, above the left and upper
 * neighbours and at least the right and lower ones, zero outside the ROI.
 *
 *   hl_circle_table_kernel -- the circles' offsets, once a handle.
 *   hl_edge_bits_kernel   -- the edge map: a bit a pixel (pixel == 255).
 *   hl_circle_bits_kernel -- a CTA a (tile, radius), largest radius first.
 *
 * The work depends on the radii and the image's size, less what cannot pass the
 * threshold: circles of fewer offsets, tiles and warps' cells with fewer edge pixels
 * in reach.  Voting point by point (hl_circle_tile_kernel) is bound by bank conflicts
 * of its shared-memory atomics, by halos (half again as many points) and by how
 * unevenly the points lie; it stays for larger radii.
 *
 * Bound by the integer pipe, about 16 operations an offset and 128 cells: ten of
 * the adders, four funnel shifts, an address.  1024 x 1024, radii 5 to 50: 67 us
 * (125 us by points); 16 pieces of 256 x 256: 86 us (136 us).  Shifts by
 * multiplication instead (the high and low products of the neighbouring words on
 * the multiply pipe) 81 and 118 us.  Votes in an order of offsets that visits 32
 * banks at a time, one point a warp: 140 us, as a circle's offsets load the banks
 * unevenly.
 */
#include <algorithm>

#include "hl_internal.h"
#include "hl_device.cuh"

#define FULL 0xffffffffu
#define CB_THREADS 256
#define CB_STRIDE (CB_THREADS + 8)   /* of a word of a plane in shared memory */
#define CB_PLANES 9       /* counts up to 511: HL_CIRCLE_DENSE_R has 504 offsets */
#define CB_HALO 4         /* words left and right of a tile in shared memory */
#define CB_TAB 512        /* table entries a radius */
/* A row of the shared edge map: word 4 q + m at CB_Q m + q, so that threads on
 * consecutive units read consecutive words whatever the column distance. */
#define CB_Q 10
/* offsets that the walk gives twice: a radius's four on the axes */
#define CB_TWICE 4

/* ---- the offsets ---------------------------------------------------------- */

/* The offsets of the radii 0 .. HL_CIRCLE_DENSE_R, a CTA a radius, sorted by
 * columns and then rows: the row distance << 16, the group << 8 (32 column
 * distances, the first from -96) and the distance in the group.  A column's
 * offsets come in pairs of rows +-i, so a group has an even number of them and two
 * neighbours of an even place are of one group.  Made once a handle, by rank: the
 * entries below an entry are counted.  Latency only.  Sorting the 22 K entries on the
 * host took 1.16 ms: the first call of a new handle, 1024 x 1024, radii 5 to 50, is
 * 200 us instead of 1346. */
__global__ void __launch_bounds__(CB_TAB) hl_circle_table_kernel(int *table)
{
    __shared__ int s_y[CB_TAB / 8], s_key[CB_TAB], s_m;
    const int tid = threadIdx.x, r = blockIdx.x;
    if (tid == 0) {   /* the walk, okano_3_0/HoughCircle.cu:214-243 */
        int m = 0;
        for (int y = r, d = 3 - 2 * r; m < y && m < CB_TAB / 8; m++) {
            s_y[m] = y;
            const bool up = d < y;
            d += up ? 4 * m + 6 : 4 * (m - y) + 10;
            y -= up ? 0 : 1;
        }
        s_m = m;
    }
    __syncthreads();
    const int n = 8 * s_m;
    int row = 0, col = 0, key = 0;
    if (tid < n) {
        const int x = tid >> 3, y = s_y[x];
        row = (tid & 1 ? x : y) * (tid & 2 ? -1 : 1);
        col = (tid & 1 ? y : x) * (tid & 4 ? -1 : 1);
        key = ((col + 128) * 256 + row + 128) * CB_TAB + tid;   /* no two alike */
        s_key[tid] = key;
    }
    __syncthreads();
    if (tid < n) {
        int rank = 0;
        for (int i = 0; i < n; i++)
            rank += s_key[i] < key;
        table[r * CB_TAB + rank] =
            (int)((unsigned)row << 16) | (((col + 96) >> 5) << 8) | (col & 31);
    }
    if (tid == 0)
        table[(HL_CIRCLE_DENSE_R + 1) * CB_TAB + r] = n;
}

/* ---- the edge map --------------------------------------------------------- */

__global__ void __launch_bounds__(256)
hl_edge_bits_kernel(const hl_circle_bits_img *imgs, hl_circle_bits_img img0, int nimg)
{
    hl_pdl_begin();
    const int blk = blockIdx.x;
    int lo = 0, hi = nimg - 1;
    while (imgs && lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (imgs[mid].blk_base <= blk)
            lo = mid;
        else
            hi = mid - 1;
    }
    const hl_circle_bits_img im = imgs ? imgs[lo] : img0;
    const long long i = (long long)(blk - im.blk_base) * 256 + threadIdx.x;
    if (i >= (long long)im.h * im.pitch)
        return;
    const int y = (int)(i / im.pitch), x = 32 * (int)(i % im.pitch);
    uint32_t m = 0;
    if (x < im.w) {
        const uint8_t *p = im.roi.base + (size_t)y * (size_t)im.roi.pitch + x;
        if (x + 32 <= im.w && (((uintptr_t)p) & 15u) == 0) {
            const uint4 *q = reinterpret_cast<const uint4 *>(p);
            m = ff_mask16(__ldcs(q)) | (ff_mask16(__ldcs(q + 1)) << 16);
        } else {
            const int n = min(32, im.w - x);
            for (int b = 0; b < n; b++)
                m |= (uint32_t)(p[b] == 255) << b;
        }
    }
    im.bits[i] = m;
}

/* ---- votes and local maxima ------------------------------------------------ */

/* words a row of the shared edge map: four pieces of CB_Q, and equal to the units
 * modulo 32 */
__host__ __device__ static inline int cb_pitch(int twu)
{
    return twu == 8 ? 4 * CB_Q : 64 + twu;
}

/* sum = sum + a + b, the carries returned */
__device__ __forceinline__ uint32_t cb_add(uint32_t &sum, uint32_t a, uint32_t b)
{
    const uint32_t c = (sum & a) | (sum & b) | (a & b);
    sum ^= a ^ b;
    return c;
}

/* one more plane of a bitwise comparison of two numbers, from the lowest: a > b,
 * or equal so far and gt */
__device__ __forceinline__ uint32_t cb_gt(uint32_t gt, uint32_t a, uint32_t b)
{
    return (a & ~b) | (gt & ~(a ^ b));
}

/* the count at relative cell (x, y) of the shared edge map, offset by offset */
__device__ __noinline__ int cb_count_at(const int2 *tab, const uint32_t *grp, int n,
                                        const uint32_t *e, int pitch, int x, int y)
{
    int v = 0;
    for (int j = 0; j < n; j++) {
        const int2 t = tab[j];
        const int k = (grp[j >> 3] >> (8 * ((j >> 1) & 3))) & 255;
        const int xx = x + 32 * (k - 3) + t.y, w = xx >> 5;
        v += (e[y * pitch + t.x / 4 + CB_Q * (w & 3) + (w >> 2)] >> (xx & 31)) & 1u;
    }
    return v;
}

/* The unit's four words at the distances of two entries of column group K (their
 * words, whole and shifted): five words each, at fixed places from the row's. */
template <int K>
__device__ __forceinline__ void cb_take(const uint32_t *mine, const int4 &e, uint32_t x[2][4])
{
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint32_t *q = reinterpret_cast<const uint32_t *>(
            reinterpret_cast<const char *>(mine) + (h ? e.z : e.x));
        uint32_t w[5];
#pragma unroll
        for (int i = 0; i < 5; i++)
            w[i] = q[CB_Q * ((K + 1 + i) & 3) + ((K + 1 + i) >> 2)];
#pragma unroll
        for (int i = 0; i < 4; i++)
            x[h][i] = __funnelshift_rc(w[i], w[i + 1], h ? e.w : e.y);
    }
}

/* The edge pixels that a unit's cells can count, by rows: pre[u (nrow + 1) + y] are
 * those of the rows below y of the shared edge map within hw words left and right of
 * unit u.  All threads. */
__device__ __noinline__ void cb_reach(int *pre, const uint32_t *e, int pitch, int twu, int nrow,
                                      int hw)
{
    for (int i = threadIdx.x; i < twu * nrow; i += CB_THREADS) {
        const int y = i / twu, u = i - y * twu;
        int c = 0;
        for (int w = CB_HALO + 4 * u - hw; w < CB_HALO + 4 * u + 4 + hw; w++)
            c += __popc(e[y * pitch + CB_Q * (w & 3) + (w >> 2)]);
        pre[u * (nrow + 1) + y + 1] = c;
    }
    __syncthreads();
    const int u = threadIdx.x >> 5, lane = threadIdx.x & 31;   /* a warp a unit */
    if (u < twu) {
        int *p = pre + u * (nrow + 1), sum = 0;
        for (int y0 = 0; y0 < nrow; y0 += 32) {
            int incl = y0 + lane < nrow ? p[y0 + lane + 1] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(FULL, incl, o);
                if (lane >= o)
                    incl += t;
            }
            if (y0 + lane < nrow)
                p[y0 + lane + 1] = sum + incl;
            sum += __shfl_sync(FULL, incl, 31);
        }
        if (lane == 0)
            p[0] = 0;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(CB_THREADS, 3)
hl_circle_bits_kernel(hl_circle_bits_args a)
{
    __shared__ __align__(16) int s_np[CB_THREADS / 32];
    extern __shared__ __align__(16) uint32_t cb_smem[];
    int2 *s_tab = reinterpret_cast<int2 *>(cb_smem);
    uint32_t *s_grp = cb_smem + 2 * CB_TAB;
    uint32_t *s_e = s_grp + CB_TAB / 8;        /* the edge map ... */
    uint32_t *s_p = s_e;                       /* ... then [plane][word][thread] */
    const int tid = threadIdx.x;
    hl_pdl_begin();
    long long rel = blockIdx.x;
    int lo = 0, hi = a.nimg - 1;
    while (a.imgs && lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (a.imgs[mid].cta_base <= rel)
            lo = mid;
        else
            hi = mid - 1;
    }
    const hl_circle_bits_img im = a.imgs ? a.imgs[lo] : a.img0;
    rel -= im.cta_base;
    const int ntile = im.ntx * im.nty;
    const int z = a.nr - 1 - (int)(rel / ntile), tile = (int)(rel % ntile);
    const int r = a.rmin + z;
    const int n = a.count[r];
    /* Only counts above the threshold are asked for: a circle, a tile or (below) a
     * warp's cells that cannot reach one are done.  1024 x 1024, radii 60 to 89,
     * threshold 178, 0.05% / 0.2% edge pixels: 37 / 49 us a call (147 / 147 without,
     * 111 / 123 by points). */
    if (!a.acc && n <= a.threshold)
        return;
    /* the tile: twu units of four words a row, rows rows; a thread a unit */
    const int twu = im.twu, rows = CB_THREADS / twu;
    const int w0 = (tile % im.ntx) * 4 * twu, y0 = (tile / im.ntx) * rows;
    const int u = tid % twu, row = tid / twu;
    const bool live = row < rows && y0 + row < im.h;
    /* the edge map around it, r + 1 rows and CB_HALO words on each side; a row's
     * pitch puts the words that a warp's threads read into different banks */
    const int pitch = cb_pitch(twu);
    const int nrow = rows + 2 * (r + 1), nq = twu + 2;   /* 16-byte pieces a row */
    int np = 0;
    for (int i = tid; i < nrow * nq; i += CB_THREADS) {
        const int yy = i / nq, q = i - yy * nq;
        const int y = y0 - r - 1 + yy, w = w0 - CB_HALO + 4 * q;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (y >= 0 && y < im.h && w >= 0 && w < im.pitch)
            v = *reinterpret_cast<const uint4 *>(im.bits + (size_t)y * im.pitch + w);
        uint32_t *d = s_e + yy * pitch + q;
        d[0] = v.x;
        d[CB_Q] = v.y;
        d[2 * CB_Q] = v.z;
        d[3 * CB_Q] = v.w;
        if (!a.acc)
            np += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
    }
    np = __reduce_add_sync(FULL, np);
    if ((tid & 31) == 0)
        s_np[tid >> 5] = np;
    /* the table's entries: the row's byte distance and the shift; four pairs'
     * groups a word */
    for (int i = tid; i < n; i += CB_THREADS) {
        const int e = a.table[CB_TAB * r + i];
        s_tab[i] = make_int2((e >> 16) * pitch * 4, e & 255);
    }
    for (int i = tid; i < n / 8; i += CB_THREADS) {
        uint32_t g = 0;
        for (int q = 0; q < 4; q++)
            g |= (uint32_t)((a.table[CB_TAB * r + 8 * i + 2 * q] >> 8) & 255) << (8 * q);
        s_grp[i] = g;
    }
    __syncthreads();
    bool reach = live;
    if (!a.acc) {
        static_assert(CB_THREADS == 256, "eight warps");
        const int4 p0 = reinterpret_cast<const int4 *>(s_np)[0];
        const int4 p1 = reinterpret_cast<const int4 *>(s_np)[1];
        np = ((p0.x + p0.y) + (p0.z + p0.w)) + ((p1.x + p1.y) + (p1.z + p1.w));
        if (np + CB_TWICE <= a.threshold)
            return;
        /* worth looking closer where the pixels, spread evenly, would not do by a
         * third: else a warp has a unit that may */
        const int hw = (r + 31) >> 5;
        if ((long long)np * (2 * r + 1) * (4 + 2 * hw) * 4 <=
            (long long)a.threshold * nrow * 4 * nq * 3) {
            int *s_pre = reinterpret_cast<int *>(s_e + nrow * pitch);
            cb_reach(s_pre, s_e, pitch, twu, nrow, hw);
            const int *p = s_pre + u * (nrow + 1) + row;
            reach = live && p[2 * r + 2] - p[1] + CB_TWICE > a.threshold;
        }
    }

    uint32_t P[CB_PLANES][4], pend[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        pend[i] = 0;
#pragma unroll
        for (int p = 0; p < CB_PLANES; p++)
            P[p][i] = 0;
    }
    if (__any_sync(FULL, reach) && live) {
        const uint32_t *mine = s_e + (row + r + 1) * pitch + u;
        for (int j = 0; j < n; j += 8) {
            uint32_t c2[4], c4[4];
            const uint32_t grp = s_grp[j >> 3];
#pragma unroll
            for (int t = 1; t < 8; t += 2) {
                /* two entries of a group (a radius has a multiple of eight) */
                uint32_t x[2][4];
                const int4 e = *reinterpret_cast<const int4 *>(s_tab + j + t - 1);
                switch ((grp >> (4 * (t - 1))) & 255) {
                case 0: cb_take<0>(mine, e, x); break;
                case 1: cb_take<1>(mine, e, x); break;
                case 2: cb_take<2>(mine, e, x); break;
                case 3: cb_take<3>(mine, e, x); break;
                case 4: cb_take<4>(mine, e, x); break;
                default: cb_take<5>(mine, e, x); break;
                }
                /* carry-save: pairs into plane 0, fours into 1, eights into 2 */
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint32_t c = cb_add(P[0][i], x[0][i], x[1][i]);
                    if (t == 1 || t == 5) {
                        c2[i] = c;
                    } else {
                        const uint32_t d = cb_add(P[1][i], c2[i], c);
                        if (t == 3) {
                            c4[i] = d;
                        } else {
                            uint32_t f = cb_add(P[2][i], c4[i], d);
                            /* every other eight waits for the next */
                            if ((j & 8) == 0) {
                                pend[i] = f;
                            } else {
                                f = cb_add(P[3][i], pend[i], f);
                                pend[i] = 0;
#pragma unroll
                                for (int p = 4; p < CB_PLANES; p++) {
                                    const uint32_t g = P[p][i] & f;
                                    P[p][i] ^= f;
                                    f = g;
                                }
                            }
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            uint32_t f = pend[i];
            /* cells outside the ROI are not counted */
            const int left = im.w - 32 * (w0 + 4 * u + i);
            const uint32_t in = left >= 32 ? FULL : (left <= 0 ? 0u : (1u << left) - 1u);
#pragma unroll
            for (int p = 3; p < CB_PLANES; p++) {
                const uint32_t g = P[p][i] & f;
                P[p][i] ^= f;
                f = g;
            }
#pragma unroll
            for (int p = 0; p < CB_PLANES; p++)
                P[p][i] &= in;
        }
    }

    /* the cells above the threshold */
    uint32_t G[4] = {0, 0, 0, 0};
    if (a.keys && a.threshold < (1 << CB_PLANES)) {
#pragma unroll
        for (int p = 0; p < CB_PLANES; p++) {
            const uint32_t t = (a.threshold >> p) & 1 ? FULL : 0u;
#pragma unroll
            for (int i = 0; i < 4; i++)
                G[i] = cb_gt(G[i], P[p][i], t);
        }
    }
    const int y = y0 + row;
    const bool up = row > 0, down = row + 1 < rows;
    /* neighbours in another tile: counted here, cell by cell */
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int x = 32 * (w0 + 4 * u + i);
        const bool west = i > 0 || u > 0, east = i < 3 || u + 1 < twu;
        uint32_t edge = (!up && y > 0) || (!down && y + 1 < im.h) ? G[i] : 0u;
        edge |= G[i] & ((!west && x > 0 ? 1u : 0u) | (!east && x + 32 < im.w ? 0x80000000u : 0u));
        while (edge) {
            const int b = __ffs(edge) - 1;
            edge &= edge - 1;
            int v = 0;
#pragma unroll
            for (int p = 0; p < CB_PLANES; p++)
                v |= (int)((P[p][i] >> b) & 1u) << p;
            const int ex = 32 * (CB_HALO + 4 * u + i) + b, ey = row + r + 1;
            bool ok = true;
            if (!up && y > 0)
                ok = ok && v > cb_count_at(s_tab, s_grp, n, s_e, pitch, ex, ey - 1);
            if (!down && y + 1 < im.h)
                ok = ok && v >= cb_count_at(s_tab, s_grp, n, s_e, pitch, ex, ey + 1);
            if (b == 0 && !west && x > 0)
                ok = ok && v > cb_count_at(s_tab, s_grp, n, s_e, pitch, ex - 1, ey);
            if (b == 31 && !east && x + 32 < im.w)
                ok = ok && v >= cb_count_at(s_tab, s_grp, n, s_e, pitch, ex + 1, ey);
            if (!ok)
                G[i] &= ~(1u << b);
        }
    }
    const bool any = (G[0] | G[1] | G[2] | G[3]) != 0;
    if (!__syncthreads_or(any) && !a.acc)
        return;
    /* the edge map is no longer read: the planes take its place */
#pragma unroll
    for (int p = 0; p < CB_PLANES; p++)
#pragma unroll
        for (int i = 0; i < 4; i++)
            s_p[(4 * p + i) * CB_STRIDE + tid] = P[p][i];
    __syncthreads();
    if (a.acc) {   /* the counts, four cells of a word a thread */
        for (int k = tid; k < 32 * twu * rows; k += CB_THREADS) {
            const int yy = k / (32 * twu), c = k - yy * 32 * twu;
            const uint32_t *q = s_p + ((c >> 3) & 3) * CB_STRIDE + yy * twu + (c >> 5);
            const int sh = 4 * (c & 7);
            /* four bits to the low bits of four bytes; the ninth plane apart */
            uint32_t v = 0;
#pragma unroll
            for (int p = 0; p < 8; p++)
                v |= ((((q[4 * p * CB_STRIDE] >> sh) & 15u) * 0x00204081u) & 0x01010101u) << p;
            const uint32_t top = q[4 * 8 * CB_STRIDE] >> sh;
            const int x = 32 * w0 + 4 * c;
            if (y0 + yy < im.h) {
                int32_t *d = a.acc + ((size_t)z * im.h + y0 + yy) * im.w + x;
                const int4 o = make_int4((int)((v & 255u) | ((top & 1u) << 8)),
                                         (int)(((v >> 8) & 255u) | ((top & 2u) << 7)),
                                         (int)(((v >> 16) & 255u) | ((top & 4u) << 6)),
                                         (int)((v >> 24) | ((top & 8u) << 5)));
                if (x + 4 <= im.w && (((uintptr_t)d) & 15u) == 0) {
                    *reinterpret_cast<int4 *>(d) = o;
                } else {
                    if (x < im.w)
                        d[0] = o.x;
                    if (x + 1 < im.w)
                        d[1] = o.y;
                    if (x + 2 < im.w)
                        d[2] = o.z;
                    if (x + 3 < im.w)
                        d[3] = o.w;
                }
            }
        }
    }
    if (!any)
        return;
    int found = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (!G[i])
            continue;
        uint32_t gw = 0, gn = 0, ge = FULL, gs = FULL;
#pragma unroll
        for (int p = 0; p < CB_PLANES; p++) {
            const uint32_t v = P[p][i];
            uint32_t l = 0, rr = 0;
            if (i > 0)
                l = P[p][i > 0 ? i - 1 : 0];
            else if (u > 0)
                l = s_p[(4 * p + 3) * CB_STRIDE + tid - 1];
            if (i < 3)
                rr = P[p][i < 3 ? i + 1 : 3];
            else if (u + 1 < twu)
                rr = s_p[4 * p * CB_STRIDE + tid + 1];
            gw = cb_gt(gw, v, (v << 1) | (l >> 31));
            ge = cb_gt(ge, v, (v >> 1) | (rr << 31));
            gn = cb_gt(gn, v, up ? s_p[(4 * p + i) * CB_STRIDE + tid - twu] : 0u);
            gs = cb_gt(gs, v, down ? s_p[(4 * p + i) * CB_STRIDE + tid + twu] : 0u);
        }
        G[i] &= gw & gn & ge & gs;
        found += __popc(G[i]);
    }
    if (!found)
        return;
    int *ncand = a.imgs ? im.ncand : a.ncand;
    unsigned long long *keys = a.imgs ? im.keys : a.keys;
    int *status = a.imgs ? im.ncand + 1 : a.status;
    int pos = atomicAdd(ncand, found);
#pragma unroll
    for (int i = 0; i < 4; i++)
        for (uint32_t m = G[i]; m; m &= m - 1) {
            const int b = __ffs(m) - 1;
            unsigned v = 0;
#pragma unroll
            for (int p = 0; p < CB_PLANES; p++)
                v |= ((P[p][i] >> b) & 1u) << p;
            const unsigned idx =
                (unsigned)(((size_t)z * im.h + y) * im.w + 32 * (w0 + 4 * u + i) + b);
            if (pos < a.cap)
                keys[pos] = ((unsigned long long)v << 32) | (unsigned)(~idx);
            else
                atomicOr(status, HL_ST_CAND_OVERFLOW);
            pos++;
        }
}

/* ---- host ------------------------------------------------------------------ */

/* table: CB_TAB entries a radius, then a count a radius */
size_t hl_circle_table_bytes(void)
{
    return (HL_CIRCLE_DENSE_R + 1) * (CB_TAB + 1) * sizeof(int);
}

cudaError_t hl_launch_circle_table(int *table, cudaStream_t s)
{
    hl_circle_table_kernel<<<HL_CIRCLE_DENSE_R + 1, CB_TAB, 0, s>>>(table);
    return cudaGetLastError();
}

/* the tiles of a w x h image: sets its pitch, twu, ntx and nty */
void hl_circle_bits_tiles(hl_circle_bits_img *im)
{
    const int words = (im->w + 31) / 32;
    im->pitch = (words + 3) & ~3;
    im->ntx = (words + 31) / 32;
    im->twu = ((words + im->ntx - 1) / im->ntx + 3) / 4;
    im->ntx = (words + 4 * im->twu - 1) / (4 * im->twu);
    const int rows = CB_THREADS / im->twu;
    im->nty = (im->h + rows - 1) / rows;
}

cudaError_t hl_launch_edge_bits(const hl_circle_bits_img *dev, const hl_circle_bits_img *im0,
                                int nimg, long long blocks, cudaStream_t s)
{
    if (blocks <= 0 || blocks > 0x7fffffffLL)
        return cudaErrorInvalidConfiguration;
    return hl_launch_pdl(hl_edge_bits_kernel, dim3((unsigned)blocks), dim3(256), 0, s, false, dev,
                         *im0, nimg);
}

/* twu_min: the narrowest tile's units (the shared edge map is tallest there) */
cudaError_t hl_launch_circle_bits(const hl_circle_bits_args *a, long long ctas, int twu_min,
                                  cudaStream_t s)
{
    size_t map = 0;
    for (int twu = twu_min; twu <= 8; twu++) {
        const size_t rows = CB_THREADS / twu + 2 * (a->rmin + a->nr);
        /* and cb_reach's sums behind it */
        map = std::max(map, rows * (size_t)cb_pitch(twu) + twu * (rows + 1));
    }
    map = std::max(map, (size_t)CB_PLANES * 4 * CB_STRIDE);
    const size_t smem = sizeof(uint32_t) * (2 * CB_TAB + CB_TAB / 8 + map);
    const cudaError_t e = cudaFuncSetAttribute(
        hl_circle_bits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess)
        return e;
    if (ctas <= 0 || ctas > 0x7fffffffLL)
        return cudaErrorInvalidConfiguration;
    return hl_launch_pdl(hl_circle_bits_kernel, dim3((unsigned)ctas), dim3(CB_THREADS), smem, s,
                         false, *a);
}
