/*
 * hl_band.h -- how the segments of a sliding vote item share out a row of
 * compaction tiles.  Plain C, so that the partition can be checked on the CPU.
 */
#ifndef HL_BAND_H
#define HL_BAND_H

#include <math.h>

#ifdef __CUDACC__
#define HL_BAND_FN __host__ __device__ __forceinline__
#else
#define HL_BAND_FN static inline
#endif

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

#endif
