/*
 * hl_band.h -- which compaction tiles of a row a vote item takes: the segments of a
 * sliding item share them out, an item of one rho window takes those that may reach
 * it.  Plain C, so that both can be checked on the CPU.
 */
#ifndef HL_BAND_H
#define HL_BAND_H

#include <math.h>

#ifdef __CUDACC__
#define HL_BAND_FN __host__ __device__ __forceinline__
#else
#define HL_BAND_FN static inline
#endif

#define HL_BAND_TILE_W 128   /* HL_TILE_W */

/* The first tile past edge j of nseg segments in a row of txn tiles whose centres
 * lie, at the slice's middle theta, yk from the image's centre line plus 1 / icm a
 * tile (x0: the first tile's centre, in tiles before the image's centre; cm has
 * icm's sign).  Edges 0 and nseg are the row's ends.  Segment j and segment j + 1
 * meet at edge j + 1, one number whichever of them asks: an edge computed from the
 * other one's differs in its last bits, and a tile whose centre lies that close
 * would be voted twice or not at all.  yk must be a rounded value (on the device
 * __fmul_rn's), so that no use fuses its product with the subtraction. */
HL_BAND_FN int hl_band_edge(int j, int nseg, int adv, float half, float yk, float cm, float icm,
                            float x0, int txn)
{
    if (j <= 0 || j >= nseg)
        return (j <= 0) == (cm > 0.0f) ? 0 : txn;
    const float e = ceilf(fmaf((float)(j * adv) - half - yk, icm, x0));
    return (int)fminf(fmaxf(e, 0.0f), (float)txn);
}

/* segment j's tiles of the row: [*ta, *tb) */
HL_BAND_FN void hl_band_tiles(int j, int nseg, int adv, float half, float yk, float cm, float icm,
                              float x0, int txn, int *ta, int *tb)
{
    const int e0 = hl_band_edge(j, nseg, adv, half, yk, cm, icm, x0, txn);
    const int e1 = hl_band_edge(j + 1, nseg, adv, half, yk, cm, icm, x0, txn);
    *ta = cm > 0.0f ? e0 : e1;
    *tb = cm > 0.0f ? e1 : e0;
}

/* p X <= q for the tile centres X = 128 i + x1 of a row: narrows the tiles [*ta,
 * *tb).  A p below 1e-5 changes p X by less than a pixel over the largest image. */
HL_BAND_FN void hl_band_half_line(float p, float q, float x1, int *ta, int *tb)
{
    if (fabsf(p) < 1.0e-5f) {
        if (q < 0.0f)
            *tb = *ta;
        return;
    }
    const float e = (q / p - x1) * (1.0f / HL_BAND_TILE_W);
    if (p > 0.0f)
        *tb = (int)fminf((float)*tb, fmaxf(floorf(e + 0.01f) + 1.0f, (float)*ta));
    else
        *ta = (int)fmaxf((float)*ta, fminf(ceilf(e - 0.01f), (float)*tb));
}

/* The tiles [*ta, *tb) of a row of txn that may hold votes of a window, on one side
 * (0 left, 1 right) of where the row's distance along the middle angle's lines
 * changes sign.  A tile's centre is (X, Y) from the image's; u = X c + Y s is its
 * distance across the lines, v = Y c - X s along them (c, s: the middle theta's).
 * Over the slice u changes by tang |v| at most, and by what lo and hi, the window's
 * ends in pixels from the image's centre, have been moved outwards for (what a tile
 * reaches from its centre, the curvature over the slice, rounding).  On one side |v| is linear in X,
 * so u - tang |v| <= hi and u + tang |v| >= lo are two half lines. */
HL_BAND_FN void hl_band_window(int side, float lo, float hi, float tang, float c, float s,
                               float x1, float y, int txn, int *ta, int *tb)
{
    const float b = side ? -tang : tang;   /* tang |v| = b v */
    int turn = y * c >= 0.0f ? txn : 0;    /* the first tile with v < 0 */
    if (s > 1.0e-6f)
        turn = (int)fminf(fmaxf(floorf((y * c / s - x1) * (1.0f / HL_BAND_TILE_W)) + 1.0f, 0.0f),
                          (float)txn);
    *ta = side ? turn : 0;
    *tb = side ? txn : turn;
    hl_band_half_line(c + b * s, hi - y * (s - b * c), x1, ta, tb);
    hl_band_half_line(b * s - c, y * (s + b * c) - lo, x1, ta, tb);
}

#endif
