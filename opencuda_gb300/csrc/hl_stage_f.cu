/*
 * hl_stage_f.cu -- the entry points either side of the plain path:
 *
 *   hl_draw_kernel      houghLineImg's line rendering (okano_3_0/HoughLine.cu:
 *                       216-249): output pixel (c, r) of the ROI becomes 255
 *                       when (int)(fl(c*cos a) + fl(r*sin a)) equals a line's
 *                       distance.  The rounded rho is monotone along a column
 *                       and along a row, so a line's pixels in one column (or
 *                       row, whichever it crosses more steeply) are one short
 *                       run: a thread takes one column of one line, estimates
 *                       the run and tests the few pixels it may hold with the
 *                       exact rule.  Work grows with the lines' pixels, not
 *                       with image pixels times lines: 32 lines of 2048 x 2048
 *                       take 3.9 us, 50.5 when every pixel tried every line.
 *   hl_real_line_kernel realLine's segment check (:252-284): edge pixels of the
 *                       segment's bounding box (grown by delta) within delta
 *                       of the segment are counted.  Only the box is
 *                       launched, not the whole image.
 */
#include "hl_internal.h"

#include <math.h>

#include <algorithm>

#define FULL 0xffffffffu
#define DRAW_THREADS 128

/* rho of pixel (c, r), okano_3_0/HoughLine.cu:238-240 */
__device__ __forceinline__ int draw_rho(int c, int r, float cs, float sn, float irho, int unit)
{
    float x = __fmul_rn((float)c, cs);
    float y = __fmul_rn((float)r, sn);
    if (!unit) {
        x = __fmul_rn(x, irho);
        y = __fmul_rn(y, irho);
    }
    return __float2int_rz(__fadd_rn(x, y));
}

__global__ void __launch_bounds__(DRAW_THREADS)
hl_draw_kernel(uint8_t *out, long pitch, int w, int h, const hl_line *lines,
               const hl_result_hdr *hdr, float irho, int unit)
{
    hl_pdl_begin();
    /* the lines of a result block: as many as were found, none after an error */
    if (hdr && ((int)blockIdx.y >= hdr->count || hdr->status != 0))
        return;
    const hl_line L = lines[blockIdx.y];
    const float cs = cosf(L.angle), sn = sinf(L.angle);
    const int d = L.distance;
    /* by column: one run of rows a column; else one run of columns a row */
    const bool by_col = fabsf(sn) >= fabsf(cs);
    const int i = blockIdx.x * DRAW_THREADS + threadIdx.x;
    const int n = by_col ? w : h, m = by_col ? h : w;
    if (i >= n)
        return;
    int j0 = 0, j1 = m - 1;
    /* truncation gives d for rho in [d, d + 1) (d > 0), (d - 1, d] (d < 0) or
     * (-1, 1); the estimate's error is far below the pixel of slack added at
     * each end (|rho| < 2^17, so a float's is below 0.02) */
    const float fixed = (float)i * (by_col ? cs : sn), slope = by_col ? sn : cs;
    const float step = 1.0f / (unit ? 1.0f : irho);
    const float lo = (float)(d > 0 ? d : d - 1) * step, hi = (float)(d < 0 ? d : d + 1) * step;
    const float a = (lo - fixed) / slope, b = (hi - fixed) / slope;
    if (fabsf(a) < 1.0e9f && fabsf(b) < 1.0e9f) {
        j0 = max(j0, (int)floorf(fminf(a, b)) - 1);
        j1 = min(j1, (int)ceilf(fmaxf(a, b)) + 1);
    } else if (a == b) {
        return;   /* both ends beyond any image on the same side */
    }
    for (int j = j0; j <= j1; j++) {
        const int c = by_col ? i : j, r = by_col ? j : i;
        if (draw_rho(c, r, cs, sn, irho, unit) == d)
            out[(size_t)r * pitch + c] = 255;
    }
}

cudaError_t hl_launch_draw(uint8_t *out, long pitch, int w, int h,
                           const hl_line *lines, int nlines, const hl_result_hdr *hdr, int derho,
                           cudaStream_t s)
{
    if (nlines <= 0 || w <= 0 || h <= 0)
        return cudaSuccess;
    /* okano_3_0/HoughLine.cu:230: float irho = 1.0f / derho, derho an int */
    const float irho = 1.0f / (float)derho;
    const unsigned gx = (unsigned)((std::max(w, h) + DRAW_THREADS - 1) / DRAW_THREADS);
    for (int first = 0; first < nlines; first += HL_DRAW_LINES) {
        const cudaError_t e =
            hl_launch_pdl(hl_draw_kernel,
                          dim3(gx, (unsigned)std::min(nlines - first, HL_DRAW_LINES)),
                          dim3(DRAW_THREADS), 0, s, false, out, pitch, w, h, lines + first, hdr,
                          irho, (int)(derho == 1));
        if (e != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

__global__ void hl_real_line_kernel(const uint8_t *img, long pitch, int w, int h,
                                    int x1, int y1, int x2, int y2, int bx0,
                                    int by0, int bx1, int by1, int delta,
                                    double len, int *count)
{
    const int cx = bx0 + blockIdx.x * blockDim.x + threadIdx.x;
    const int ry = by0 + blockIdx.y * blockDim.y + threadIdx.y;
    int hit = 0;
    if (cx <= bx1 && ry <= by1 && cx < w && ry < h && cx >= 0 && ry >= 0) {
        if (img[(size_t)ry * pitch + cx] == 255) {
            /* okano_3_0/HoughLine.cu:275: |cross| / |segment| in double,
             * stored as float, compared with the int delta */
            int cr = abs((x2 - x1) * (ry - y1) - (cx - x1) * (y2 - y1));
            float dis = __double2float_rn(__ddiv_rn((double)cr, len));
            hit = dis < (float)delta;
        }
    }
    const unsigned b = __ballot_sync(FULL, hit);
    if ((threadIdx.x & 31) == 0 && b)
        atomicAdd(count, __popc(b));
}

cudaError_t hl_launch_real_line(const uint8_t *img, long pitch, int w, int h,
                                int x1, int y1, int x2, int y2, int delta,
                                int *count, cudaStream_t s)
{
    const int xmin = min(x1, x2), xmax = max(x1, x2);
    const int ymin = min(y1, y2), ymax = max(y1, y2);
    /* okano_3_0/HoughLine.cu:266-267: cx in [xmin - delta, xmax + delta] */
    const int bx0 = max(xmin - delta, 0), bx1 = min(xmax + delta, w - 1);
    const int by0 = max(ymin - delta, 0), by1 = min(ymax + delta, h - 1);
    if (bx1 < bx0 || by1 < by0)
        return cudaSuccess;
    const double len = sqrt((double)(x2 - x1) * (x2 - x1) * 1.0 +
                            (double)(y2 - y1) * (y2 - y1));
    dim3 block(32, 8);
    dim3 grid((bx1 - bx0 + 32) / 32, (by1 - by0 + 8) / 8);
    hl_real_line_kernel<<<grid, block, 0, s>>>(img, pitch, w, h, x1, y1, x2, y2,
                                               bx0, by0, bx1, by1, delta, len,
                                               count);
    return cudaGetLastError();
}
