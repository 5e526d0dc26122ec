/*
 * hl_internal.h -- kernel argument blocks and launchers shared by the
 * translation units of libhoughline_gb300.so (not part of the C ABI).
 */
#ifndef HL_INTERNAL_H
#define HL_INTERNAL_H

#include <cuda_runtime.h>
#include <stdint.h>

#include "houghline_gb300.h"
#include "hl_circle.h"

#include <utility>

/* Compaction tiles: 128 x 32 pixels; one CTA of 256 threads reads one tile,
 * 16 pixels (one 16-byte vector) per thread. */
#define HL_TILE_W 128
#define HL_TILE_H 32
#define HL_COMPACT_THREADS 256
/* Tiles per compaction CTA (one look-back per group). */
#define HL_COMPACT_GROUP 4
/* Theta slice = one warp: lane i owns theta k0 + i. */
#define HL_SLICE 32

/* Bits of the device status word. */
#define HL_ST_LOOKBACK_TIMEOUT 0x1
#define HL_ST_CAND_OVERFLOW 0x2
#define HL_ST_RHO_OUT_OF_RANGE 0x4
#define HL_ST_MERGE_OVERFLOW 0x8
#define HL_ST_VOTE_TIMEOUT 0x10
#define HL_ST_CNN_TIMEOUT 0x20

/* Result block written by the finalize kernel (device) and copied to the
 * host in one transfer. */
typedef struct hl_result_hdr {
    int count;    /* lines written = min(survivors, linesmax) */
    int status;   /* HL_ST_* bits seen during this call */
    int ncand;    /* peaks found */
    int pad;
} hl_result_hdr;

typedef struct hl_roi {
    const uint8_t *base;  /* ROI origin */
    long pitch;
    int w, h;
} hl_roi;

/* One image of a batched compaction: its tiles occupy [tile_base, +ntiles)
 * of the batch's tile_off array, its 4-tile groups [group_base, +ngroups) of
 * the batch's group space, and its points start at pts_base of the batch's
 * point array (room for every pixel plus one pad per tile).  Prefixes and
 * tile offsets are per image: an image's groups wait only for each other. */
typedef struct hl_compact_img {
    hl_roi roi;
    int tiles_x, ntiles;
    int tile_base, group_base, ngroups;
    int pad;
    long long pts_base;
} hl_compact_img;

typedef struct hl_compact_args {
    /* one image (imgs == NULL) ... */
    hl_roi roi;
    int tiles_x, ntiles;
    /* ... or a batch: group g belongs to image group_img[g] */
    const hl_compact_img *imgs;
    const int *group_img;
    int nimg, ngroups;
    unsigned long long *tile_state;  /* [ntiles], epoch-tagged */
    unsigned int *ticket;            /* monotonically increasing counter */
    unsigned int ticket_base;        /* value of *ticket at launch */
    unsigned int epoch;              /* 1..2^30-1, distinct per launch */
    uint32_t *pts;                   /* out: packed x | y << 16, or NULL */
    float2 *pts_f2;                  /* out: (x, y) as floats, or NULL */
    int *tile_off;                   /* out: [ntiles + 1] */
    int *count;                      /* out: total points */
    int *status;
} hl_compact_args;


/* One image of a vote launch. */
typedef struct hl_vote_img {
    const float2 *pts;        /* (x, y) of every edge point, tile-major */
    const int *tile_off;      /* the image's [ntiles + 1] tile offsets */
    int ntiles, tiles_x;
    int w, h;                 /* ROI size */
    int rho_min, R;
    int threshold;            /* peak threshold: bins above it are noted */
    int pad;
    /* [R][Tp], zero at the launch: with a candidate list the bins above the
     * threshold are stored, without one every row that a vote can reach */
    int32_t *acc;
} hl_vote_img;

/* One work item of the vote: a rectangle of an image's compaction tiles (a
 * region) voted for one theta slice.  Every theta's window of rows starts at
 * the lowest rho the rectangle reaches, so `rows` of them hold every vote. */
typedef struct hl_vote_item {
    int img, slice;
    int tx, ty;               /* first tile | tiles << 16 */
    int slab;                 /* its slab's first row group in scratch; -1: the
                                 block's only item, or a whole window, or
                                 hl_vote_args.add */
    int gb[4], gn[4], go[4];  /* the slab's column groups: see hl_slab */
    /* win: a whole image's votes of one window of adv rows; column k's row 0 is
     * floor(rho of the centre at theta_k) + off0.  Tiles that may reach the window
     * are voted (hl_band_window: lo, hi, tang), every vote's row is tested.  The
     * windows of a block hold all its rows, so each is final unless its points are
     * shared out to nparts items (this one is part `part`).  nseg: groups of
     * HL_VOTE_RUNS / 2 tile rows */
    int win, part, nparts;
    float lo, hi, tang;
    /* else nseg > 1: a whole image whose range does not fit one window, voted in
     * nseg segments with the window sliding by adv rows after each: segment j
     * holds the tiles whose centre lies, at the slice's middle theta, [j adv,
     * (j + 1) adv) above -half from the image's centre; column k's row 0 is
     * floor(rho of the centre at theta_k) + off0 + j adv */
    int nseg, adv, off0;
    float half;
} hl_vote_item;

/* A slab of scratch: the counts of an item as its block's merge reads them.
 * Four groups of 8 columns; group g holds the accumulator rows [4 b[g],
 * 4 (b[g] + n[g])), which every vote of the group falls into, in row groups of
 * four, [row group][column][4 rows], 16-bit counts (64 bytes a row group) or
 * 32-bit ones (128), from row group o[g] of the slab on. */
typedef struct hl_slab {
    int at;                   /* its first row group in scratch */
    int lo, hi;               /* row groups that some column group holds */
    int pad;
    int b[4], n[4], o[4];
} hl_slab;

/* Peak candidates of a launch: every accumulator bin above its image's
 * threshold, noted as image << 32 | (row * T + theta) when its final count
 * is stored (the vote's block store, the merge of a split block); the other
 * bins stay zero.  A counter past cap means some were not noted: the peak pass
 * then scans every accumulator instead.  The counter is zero at the vote's
 * start (a batch clears it with its other counters; single images alternate
 * between two, and a call's tail clears the next one's); e == NULL: nothing is
 * noted and whole accumulators are stored. */
typedef struct hl_cand_list {
    unsigned long long *e;
    int *count;
    int cap;
    int pad;
} hl_cand_list;

typedef struct hl_vote_args {
    const hl_vote_img *imgs;  /* per image, or NULL: the one image img0 */
    hl_vote_img img0;
    const float *cosv, *sinv; /* [theta_pad] */
    int T, Tp;
    int win_rows;             /* rows of a window in shared memory */
    float irho;
    int exact;                /* |rho| may reach 2^22: convert exactly */
    int *status;
    /* persistent scheduling: items are taken in order (heaviest first) from a
     * monotonically increasing counter */
    const hl_vote_item *items;
    int nitems;
    int win;                  /* some of them are of one window each */
    unsigned *work;           /* counter */
    unsigned work_base;       /* its value at launch */
    unsigned char *scratch;   /* slabs: row groups */
    int part16;               /* slabs hold 16-bit counts (hl_part16_ok) */
    int add;                  /* no slabs: items add to the cleared accumulator */
    hl_cand_list cand;
} hl_vote_args;

/* A block (an image's theta slice) voted in several items: its accumulator
 * columns are the sum of the slabs [first, first + n) of the slab list. */
typedef struct hl_merge_block {
    int img, slice;
    int first, n;
    int lo, hi;               /* row groups that some slab holds */
} hl_merge_block;

typedef struct hl_merge_args {
    const hl_vote_img *imgs;  /* as in hl_vote_args */
    hl_vote_img img0;
    int T, Tp;
    const unsigned char *scratch;
    const hl_merge_block *blocks;
    int nblocks;
    unsigned chunks;          /* CTAs a block: 16 row groups each */
    const hl_slab *slabs;
    int part16;
    hl_cand_list cand;
} hl_merge_args;

struct hl_peak_img;

/* Can an item's counts be kept in 16 bits?  A bin of one rho bin width
 * derho (the rho-0 bin spans two, truncation toward zero) holds the pixels of
 * a strip of width <= 2 derho across the region: fewer than (2 derho + 2)
 * (w + h) of them. */
static inline int hl_part16_ok(double derho, int w, int h)
{
    return (2.0 * derho + 2.0) * ((double)w + (double)h) < 65535.0;
}

/* Tiles the allocation-free compaction entry point can serve. */
#define HL_NOALLOC_MAX_TILES 65536

/* Vote-kernel staging: points per ring slot, ring slots; tile rows of a region
 * at most (unless it spans the image's width: then its points are one run). */
#ifndef HL_VOTE_CHUNK
#define HL_VOTE_CHUNK 2048
#endif
#ifndef HL_VOTE_SLOTS
#define HL_VOTE_SLOTS 2
#endif
#define HL_VOTE_RUNS 128
/* largest rho window (rows) one CTA can hold next to its staging */
int hl_vote_max_rows(void);

/* One image of a peak pass. */
typedef struct hl_peak_img {
    const int32_t *acc;       /* [R][Tp] */
    unsigned long long *keys; /* votes << 32 | ~tight_index */
    int *ncand;
    int R, cap;
    int threshold;            /* votes must exceed it */
    int pad;
} hl_peak_img;

/* rows of an accumulator one peak-pass chunk covers (several images), int4
 * of a unit of one image's accumulator, threads of a peak-pass CTA */
#define HL_PEAK_ROWS 16
#define HL_PEAK_THREADS 256
#define HL_PEAK_LOADS 4           /* 16-byte loads in flight per thread */
#define HL_PEAK_FLAT (HL_PEAK_LOADS * HL_PEAK_THREADS)
#define HL_PEAK_CTAS_PER_SM 6

typedef struct hl_peak_args {
    const hl_peak_img *imgs;  /* per image, or NULL: the one image img0 */
    hl_peak_img img0;
    const int2 *chunks;       /* {image, first row}, HL_PEAK_ROWS rows each;
                                 NULL: unit c is int4 c * HL_PEAK_FLAT.. of
                                 img0's accumulator */
    int nchunks;
    int T, Tp;
    int *status;
    /* the bins above the threshold, noted by the vote and the merge; when
     * they all fit, only they are tested (no scan of the accumulators) */
    hl_cand_list cand;
} hl_peak_args;

/* One image of a finalize launch (one CTA per image). */
typedef struct hl_final_img {
    const unsigned long long *keys;
    int *ncand;               /* read, then reset to 0 for the next call */
    int cap;
    int rho_min, ref_numrho;
    int pad;
    hl_line *lines;           /* out: [linesmax] */
    int *count_out;           /* out: lines written, or NULL */
} hl_final_img;

typedef struct hl_final_args {
    const hl_final_img *imgs; /* per image (CTA), or NULL: the one image img0 */
    hl_final_img img0;
    int T;
    double detheta;
    int thresdis;
    float thresang;
    int linesmax;
    hl_result_hdr *hdr;       /* out (one image), or NULL */
    int *status;              /* read; reset to 0 when hdr is set */
    /* the bins that the vote stored above the threshold, cleared again (the
     * whole accumulator when they did not all fit the list); e NULL: none */
    hl_cand_list clear;
    const hl_peak_img *clear_imgs;   /* per image, or NULL: acc */
    int32_t *acc;                    /* acc_ints of them */
    long long acc_ints;
    int Tp;
    int *cand_count;          /* another call's candidate counter, reset to 0
                                 for the next one (or NULL) */
} hl_final_args;

/* The whole plain path of one small image in one cluster launch (see
 * hl_small_kernel): usable when Tp / 32 <= HL_SMALL_MAX_CTAS and the R x 32
 * accumulator slice plus its dump row fit one CTA's shared memory. */
#define HL_SMALL_MAX_CTAS 8
typedef struct hl_small_args {
    hl_roi roi;
    float2 *pts;              /* w * h entries of scratch (global) */
    const float *cosv, *sinv; /* [Tp] */
    int T, Tp, R, rho_min;
    float irho;
    int threshold;
    hl_final_args fin;        /* keys, counters, result records */
    float scale;              /* (float)(1 / (T + 2)), the reference decode */
} hl_small_args;
int hl_small_fits(int T, int Tp, int R);
cudaError_t hl_launch_small(const hl_small_args *a, cudaStream_t s);

/* launchers (return cudaGetLastError() after the launch) */
cudaError_t hl_launch_trig(float *cosv, float *sinv, int T, int Tp,
                           double detheta, cudaStream_t s);
#ifdef __CUDACC__
/* Programmatic dependent launch: the pipeline's kernels are launched with
 * programmatic stream serialization, so a kernel's grid can be set up while
 * its predecessor drains.  Each kernel waits for its predecessor's completion
 * (and memory) before it touches global memory, then lets its own successor
 * launch.  Both are no-ops for a kernel launched the ordinary way. */
__device__ __forceinline__ void hl_pdl_begin()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

/* launch `kernel` with programmatic stream serialization (and, if coop, as a
 * cooperative launch) */
template <typename... Params, typename... Args>
static inline cudaError_t hl_launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block,
                                        size_t smem, cudaStream_t s, bool coop,
                                        Args &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeCooperative;
    at[1].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = coop ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
#endif
/* HoughCircle (hl_circle_bits.cu, hl_circle.cu) */
/* Radii up to this are counted on bit planes (nine of them, three words left and
 * right), larger ones vote point by point.  1024 x 1024, the whole call against the
 * same by points, threshold 100 or twice the radius: radii 5 to 50, 5% edge pixels 97
 * against 320 us, 1% 87 against 135, 0.05% 38 against 99; 60 to 89, 1% 147 against
 * 209, 0.05% 37 against 111.  Slower where few edge pixels meet a low threshold or the
 * whole accumulator is asked for: 60 to 89, 0.05%, threshold 30 135 against 111, the
 * accumulator 184 against 150. */
#define HL_CIRCLE_DENSE_R 89
/* One image's edge map and its tiles.  A call's only image has bases 0. */
typedef struct hl_circle_bits_img {
    hl_roi roi;
    uint32_t *bits;           /* [h][pitch], bit b of word x / 32 is pixel x */
    int w, h;
    int pitch;                /* words, a multiple of 4 */
    int ntx, nty, twu;        /* tiles; 16-byte units of a tile's row, 1 .. 8 */
    int blk_base;             /* first CTA of hl_edge_bits_kernel: 256 words each */
    long long cta_base;       /* first CTA of hl_circle_bits_kernel */
    unsigned long long *keys; /* as in hl_circle_img */
    int *ncand;
} hl_circle_bits_img;
typedef struct hl_circle_bits_args {
    const hl_circle_bits_img *imgs;   /* or NULL: img0 */
    hl_circle_bits_img img0;
    int nimg;
    int rmin, nr;             /* rmin + nr - 1 <= HL_CIRCLE_DENSE_R */
    const int *table, *count; /* hl_circle_table_kernel */
    int32_t *acc;             /* [nr][h][w], or NULL */
    int threshold;
    unsigned long long *keys; /* one image: votes << 32 | ~index, or NULL */
    int *ncand;
    int cap;
    int *status;
} hl_circle_bits_args;
size_t hl_circle_table_bytes(void);
cudaError_t hl_launch_circle_table(int *table, cudaStream_t s);
void hl_circle_bits_tiles(hl_circle_bits_img *im);
cudaError_t hl_launch_edge_bits(const hl_circle_bits_img *dev, const hl_circle_bits_img *im0,
                                int nimg, long long blocks, cudaStream_t s);
cudaError_t hl_launch_circle_bits(const hl_circle_bits_args *a, long long ctas, int twu_min,
                                  cudaStream_t s);
#define HL_CIRCLE_MAXCAND 4096
/* One CTA per (accumulator tile, radius): the tile and a one-cell apron are
 * counted in shared memory from the points of the halo (the compaction tiles
 * within the radius of the tile); then the interior is written to acc and/or
 * its local maxima appended to keys. */
#define HL_CIRCLE_TW 256
#define HL_CIRCLE_TH 192
/* One image of a circle batch: its points and tile offsets (the batch
 * compaction's region of the image), its ROI, its candidate keys and
 * counters, its result records, and the first CTA of its tile launch. */
typedef struct hl_circle_img {
    const float2 *pts;
    const int *tile_off;
    int ctiles_x, ctiles_y;
    int w, h;
    int ntx, nty;
    int roi_x, roi_y;
    int cta_base;
    int pad;
    unsigned long long *keys; /* [HL_CIRCLE_MAXCAND] */
    int *ncand;               /* [ncand, status] */
    hl_circle *out;
    hl_result_hdr *hdr;
} hl_circle_img;
typedef struct hl_circle_tile_args {
    /* a batch: the CTA's image is the last with cta_base <= blockIdx.x, and
     * its fields replace pts .. nty, keys, ncand and status below */
    const hl_circle_img *imgs;
    int nimg;
    int nctas;                /* CTAs of a batch (every image's tiles x radii) */
    const float2 *pts;        /* the compaction's points (odd tiles padded) */
    const int *tile_off;      /* [ctiles_x * ctiles_y + 1] */
    int ctiles_x, ctiles_y;   /* compaction tiles (HL_TILE_W x HL_TILE_H) */
    int w, h;                 /* ROI */
    int rmin, nr;
    int nz;                   /* the largest nz of them are voted */
    int ntx, nty;             /* accumulator tiles */
    int32_t *acc;             /* [nr][h][w], or NULL */
    int threshold;
    unsigned long long *keys; /* votes << 32 | ~index, or NULL */
    int *ncand;
    int cap;
    int *status;
} hl_circle_tile_args;
typedef struct hl_circle_final_args {
    /* a batch: CTA i takes image i's keys, counters, ROI and outputs */
    const hl_circle_img *imgs;
    const unsigned long long *keys;
    int *ncand;
    int w, h, rmin;
    float dist_thres;
    int r_thres;
    int circlemax;
    int roi_x, roi_y;         /* added to the centres */
    hl_circle *out;
    hl_result_hdr *hdr;
    int *status;
} hl_circle_final_args;
cudaError_t hl_launch_circle_tiles(const hl_circle_tile_args *a, cudaStream_t s);
/* grid: one CTA, or nimg CTAs for a batch */
cudaError_t hl_launch_circle_final(const hl_circle_final_args *a, int nimg, cudaStream_t s);

cudaError_t hl_launch_compact(const hl_compact_args *a, cudaStream_t s);
/* one image (a->imgs == NULL) with hl_compact_persist_ctas(ntiles, sms) CTAs
 * in a cooperative launch (0: too many to be resident at once), each adding
 * one to the ticket word */
int hl_compact_persist_ctas(int ntiles, int sms);
cudaError_t hl_launch_compact_persist(const hl_compact_args *a, int nct, cudaStream_t s);
cudaError_t hl_launch_merge(const hl_merge_args *a, cudaStream_t s);
cudaError_t hl_launch_vote(const hl_vote_args *a, int threads, int grid,
                           cudaStream_t s);
size_t hl_vote_smem_bytes(int win_rows);
/* the vote over a coordinate list: clears acc, then votes */
typedef struct hl_points_args {
    const int2 *xy;
    int n;
    int x0, y0, x1, y1;       /* its bounding box */
    const float *cosv, *sinv; /* [Tp] */
    int T, Tp;
    int rho_min, R;
    int span;                 /* rows any slice's range over the box needs at most */
    int win_rows;             /* set by the launcher */
    int exact;                /* |rho| may reach 2^22: convert exactly */
    float irho;
    int32_t *acc;             /* [R][Tp] */
} hl_points_args;
cudaError_t hl_launch_vote_points(hl_points_args *a, int sms, cudaStream_t s);
cudaError_t hl_launch_peaks(const hl_peak_args *a, cudaStream_t s);
cudaError_t hl_launch_finalize(const hl_final_args *a, int nimg, cudaStream_t s);
cudaError_t hl_launch_to_tight(const int32_t *acc, int R, int T, int Tp,
                               int32_t *out, cudaStream_t s);
cudaError_t hl_launch_to_ref(const int32_t *acc, int R, int T, int Tp,
                             int rho_min, int ref_numrho, int32_t *ref,
                             cudaStream_t s);
cudaError_t hl_launch_from_tight(const int32_t *acc, int R, int T, int Tp,
                                 int32_t *out, cudaStream_t s);
/* CTAs of the bounding-box kernel at most (their partial boxes in part) */
#define HL_BBOX_CTAS 152
/* bounding box {xmin, ymin, xmax, ymax} of a list; bbox may be mapped host
 * memory, *ticket is zero before and after */
cudaError_t hl_launch_bbox(const int *xy, int n, int4 *part, unsigned *ticket, int *bbox,
                           cudaStream_t s);
/* lines of one drawing launch */
#define HL_DRAW_LINES 32768
/* hdr NULL: nlines lines; else at most HL_DRAW_LINES, and only the hdr->count
 * that were found (none after an error) */
cudaError_t hl_launch_draw(uint8_t *out, long pitch, int w, int h,
                           const hl_line *lines, int nlines, const hl_result_hdr *hdr, int derho,
                           cudaStream_t s);
cudaError_t hl_launch_real_line(const uint8_t *img, long pitch, int w, int h,
                                int x1, int y1, int x2, int y2, int delta,
                                int *count, cudaStream_t s);
cudaError_t hl_launch_atomic_bench(int iters, int *sink, cudaStream_t s,
                                   int *blocks_out, int *threads_out);

#endif
