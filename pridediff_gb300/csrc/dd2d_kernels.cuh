// Shared device code of the 2-D DD projector: layouts, the integral-form
// evaluation and the adjoint's work-item bodies (pixel gathers; the forward's
// is in dd2d_fwd.cuh).  Included by dd2d.cu (single-geometry launches) and
// dd2d_batch.cu (persistent launches over uneven instances).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include <cooperative_groups.h>

#include "../../include/pridediff_dd.h"
#include "dd_geom2d.cuh"
#include "dd_tma.cuh"

namespace dd2 {


constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kBinsPerWarp = 31;   // 32 boundaries -> 31 bins per warp pass
constexpr int kBI = 4;             // images per CTA (geometry amortised over them)
constexpr int kTile = 32;          // adjoint work item: 32 x 32 pixels
// Adjoint-map entries per walked line of a tile: the boundaries of a 32-pixel
// run plus one below it, from an even first entry (36), padded to an odd
// number of 8-byte entries so that the lanes of a warp reading 32 different
// lines' rows hit distinct shared-memory banks.
constexpr int kMapE = 37;
// One adjoint-map block (a view, a tile): kTile rows of kMapE entries {bin,
// offset}, then the kTile lines' DD-BP scales; one bulk copy moves it.
constexpr int kMapBlkBytes = kTile * kMapE * 8 + kTile * 4;

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }
__host__ __device__ inline int rs_entries(int n) { return (n + 2) & ~1; }   // n+1 float2, 16-B rows

// ---------------------------------------------------------------------------
// Workspace layout
// ---------------------------------------------------------------------------
struct PlanLayout {
    size_t views, ang, dp, bcoef, lines, dlines, axisv, amap, trange, total;
    int nl;   // line records per view = max(H, W)
};

// Adjoint map of fan beams, one block per (view, tile) in tile-major order.
// Entry e of a walked line holds its boundary e - 1 (e in 0 .. map_stride()-1
// over the line); a block keeps, for each of the tile's kTile walked lines,
// the kMapE entries from the tile's first entry (map_first()).
__host__ __device__ inline int map_stride(const dd_geom2d *g) {
    return rs_entries(g->width > g->height ? g->width : g->height);
}
// 32 x 32 tiles of the image (the adjoint's work items); tile = ty * ntx + tx
__host__ __device__ inline int tiles_x(const dd_geom2d *g) { return (g->width + 31) / 32; }
__host__ __device__ inline int tiles_n(const dd_geom2d *g) { return tiles_x(g) * ((g->height + 31) / 32); }
// First map entry a tile's block keeps.  Rows (xb views): pixels c0 .. c0+31
// have boundaries c0-1 .. c0+31, entries c0 .. c0+32.  Columns: pixels
// H-r0-32 .. H-r0-1 along the column, entries from an even index at or below
// H-r0-32 (so that 36 entries always reach H-r0).
__host__ __device__ inline int map_first(const dd_geom2d *g, int xb, int c0, int r0) {
    if (xb) return c0;
    const int lo = g->height - r0 - kTile;
    return (lo > 0 ? lo : 0) & ~1;
}

// with_map = false leaves out the adjoint map (plans that only serve the
// forward-type operators, e.g. one-shot forward calls); every other offset is
// the same either way.
inline PlanLayout plan_layout(int scan, const dd_geom2d *g, int V, bool with_map = true) {
    PlanLayout L;
    const int D = g->num_det;
    L.nl = g->height > g->width ? g->height : g->width;
    size_t o = 0;
    L.views = o; o = align_up(o + sizeof(DdView2) * (size_t)V, 256);
    L.ang = o; o = align_up(o + sizeof(float) * (size_t)V, 256);
    L.dp = o; o = align_up(o + sizeof(float) * (size_t)V * (D + 1), 256);
    L.bcoef = o; o = align_up(o + sizeof(float) * (size_t)V * (D + 1), 256);
    L.lines = o; o = align_up(o + sizeof(DdLine) * (size_t)V * L.nl, 256);
    L.dlines = o;
    if (scan == DD_SCAN_PARA) o = align_up(o + sizeof(DdLine) * (size_t)V * L.nl, 256);
    // the adjoint's view lists: those that walk rows and those that walk
    // columns ({count rows, count columns, rows' views[V], columns' views[V]})
    L.axisv = o;
    if (scan == DD_SCAN_PARA) o = align_up(o + sizeof(int) * (2 * (size_t)V + 2), 256);
    L.amap = L.trange = o;
    if (scan != DD_SCAN_PARA && with_map) {
        L.amap = o; o = align_up(o + (size_t)kMapBlkBytes * V * tiles_n(g), 256);
        L.trange = o; o = align_up(o + sizeof(int2) * (size_t)V * tiles_n(g), 256);
        L.axisv = o; o = align_up(o + sizeof(int) * (2 * (size_t)V + 2), 256);
    }
    L.total = o;
    return L;
}

struct ApplyLayout {
    size_t tabx, taby, dtab, status, total;
};

inline bool op_is_forward(int op) {
    return op == DD_OP_PROJ || op == DD_OP_BPROJ_T || op == DD_OP_BPROJ_TW;
}

inline ApplyLayout apply_layout(int op, const dd_geom2d *g, int B, int V) {
    ApplyLayout L;
    size_t o = 0;
    L.tabx = L.taby = L.dtab = 0;
    if (op_is_forward(op)) {
        // the planes of rows and columns (8 bytes a pixel hold any grouping of
        // the slices), or their prefix tables
        L.tabx = o; o = align_up(o + sizeof(float2) * (size_t)B * g->height * rs_entries(g->width), 256);
        L.taby = o; o = align_up(o + sizeof(float2) * (size_t)B * g->width * rs_entries(g->height), 256);
    } else {
        L.dtab = o; o = align_up(o + sizeof(float2) * (size_t)B * V * rs_entries(g->num_det), 256);
    }
    L.status = o; o = align_up(o + 256, 256);
    L.total = o;
    return L;
}

// ---------------------------------------------------------------------------
// Shared device pieces of the integral evaluation
// ---------------------------------------------------------------------------
// Per-piece constants K_p of one line for table `tab` (lane p < npiece).
// F(u) = K_p + dl_p S_j + r x_j on piece p (see file header).
__device__ __forceinline__ float piece_K(const DdLine &L, const float2 *tab, int lane) {
    const int np = L.h.npiece;
    float term = 0.0f;
    if (lane < np) {
        const DdPiece P = L.p[lane];
        const int first = (lane == 0) ? L.h.i0 : L.p[lane - 1].gb + 1;
        const float fv = FADD(P.Q, FMUL((float)(first - P.gb), P.dl));
        const float prevQ = (lane == 0) ? L.h.bound0 : L.p[lane - 1].Q;
        const float prevdl = (lane == 0) ? 0.0f : L.p[lane - 1].dl;
        const float2 e0 = tab[first];
        const float S1 = tab[first + 1].x;
        term = fmaf(prevdl, e0.x, fmaf(e0.y, fv - prevQ, -P.dl * S1));
    }
    for (int o = 1; o < 32; o <<= 1) {
        const float y = __shfl_up_sync(0xffffffffu, term, o);
        if (lane >= o) term += y;
    }
    return term;
}

// FBP-weight pixel centre a * pitch + shift, a an exact half-integer offset:
// one FMA rounds the exact value once.  The reference evaluates the same
// expression in FP64 and rounds that to FP32, which gives the same float
// unless the exact value lies within 2^-53 (relative) of an FP32 rounding
// boundary -- and FP64 arithmetic runs at a small fraction of the FP32 rate.
__device__ __forceinline__ float pix_centre(float a, float pitch, float shift) { return fmaf(a, pitch, shift); }

// ---------------------------------------------------------------------------
// Prefix tables in double-float arithmetic.  A sum is carried as an unevaluated
// pair hi + lo of floats (two-sum and FMA two-product are exact), about 48
// significant bits; hi of the pair is the sum rounded to FP32.  FP64 would do
// the same, but GB300 runs FP64 at a small fraction of its FP32 rate and the
// tables' scans were bound by it.
// ---------------------------------------------------------------------------
struct DdF {
    float hi, lo;
};
__device__ __forceinline__ DdF df_add(DdF a, DdF b) {
    const float s = __fadd_rn(a.hi, b.hi);
    const float v = __fsub_rn(s, a.hi);
    const float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, v)), __fsub_rn(b.hi, v));
    const float t = __fadd_rn(e, __fadd_rn(a.lo, b.lo));
    const float hi = __fadd_rn(s, t);
    return {hi, __fsub_rn(t, __fsub_rn(hi, s))};
}
__device__ __forceinline__ DdF df_prod(float a, float b) {
    const float p = __fmul_rn(a, b);
    return {p, __fmaf_rn(a, b, -p)};
}
__device__ __forceinline__ DdF df_shfl_up(DdF a, int o) {
    return {__shfl_up_sync(0xffffffffu, a.hi, o), __shfl_up_sync(0xffffffffu, a.lo, o)};
}
__device__ __forceinline__ DdF df_shfl(DdF a, int l) {
    return {__shfl_sync(0xffffffffu, a.hi, l), __shfl_sync(0xffffffffu, a.lo, l)};
}

// One warp: entries k = 0 .. n of t get (sum_{m<k} v_m, x_k) for the values
// v_k = x_k * w_k produced by val(k, &x, &w) (x = w = 0 past the end).
template <typename F>
__device__ __forceinline__ void warp_prefix_table(int n, float2 *t, int lane, F val) {
    DdF run = {0.0f, 0.0f};
    for (int k0 = 0; k0 <= n; k0 += 32) {
        const int k = k0 + lane;
        float x = 0.0f, w = 0.0f;
        if (k < n) val(k, &x, &w);
        DdF inc = df_prod(x, w);
        for (int o = 1; o < 32; o <<= 1) {
            const DdF y = df_shfl_up(inc, o);
            if (lane >= o) inc = df_add(inc, y);
        }
        DdF prev = df_shfl_up(inc, 1);
        if (lane == 0) prev = {0.0f, 0.0f};
        if (k <= n) t[k] = make_float2(df_add(run, prev).hi, x);
        run = df_add(run, df_shfl(inc, 31));
    }
}

// FBP weight of a fan-beam pixel centre (px, py) for the source (sx, sy):
// flat detector r^2 / (r - s.p / r)^2 (FanFlatDisCPU2d.cpp:693, r the
// source radius), evaluated as (r^2 / (r^2 - s.p))^2 with one fast division
// (__fdividef: within 2 ulp for these magnitudes) instead of two IEEE
// divisions; arc detector 1 / |s - p|^2 (FanArcDisCPU2d.cpp:703).  Within a
// few ulp of the reference's FP32 sequence; the forward-type and the
// adjoint-type kernels both use it, so BackProjWeighted and
// BackProjTransWeighted stay exact transposes.
template <int GEOM>
__device__ __forceinline__ float fan_fbp_weight(float sx, float sy, float px, float py, float r) {
    if (GEOM == DD_GEOM_ARC) {
        const float a = sx - px, b = sy - py;
        return __fdividef(1.0f, fmaf(a, a, b * b));
    }
    const float r2 = r * r;
    const float t = __fdividef(r2, r2 - fmaf(sx, px, sy * py));
    return t * t;
}

// The longest lines for which dd2d_fwd_shape says 4 slices and the uneven batch
// takes an instance: those of which 4 slices' prefix tables fit one CTA twice, at
// 8 warps of 31 bins.  (A limit of the interface; how many slices a CTA then
// takes is a matter of dd2d_fwd.cuh's fwd_fits.)
inline long long four_slice_bytes(bool para, int D, int npix, int cl) {
    const int n = (D + kWarps * kBinsPerWarp - 1) / (kWarps * kBinsPerWarp);
    const int npass = n <= 1 ? 1 : n <= 2 ? 2 : n <= 3 ? 3 : n <= 4 ? 4 : 8;
    const long long tabs = 2LL * kBI * rs_entries(npix) * (long long)sizeof(float2);
    const long long red = cl > 1 ? (long long)npass * kBI * kThreads * (long long)sizeof(float) : 0;
    const long long o = (para ? 4LL : 2LL) * (long long)sizeof(DdLine) + std::max(tabs, red) +
                        kBI * 32 * (long long)sizeof(float) + ((D + 1 + 3) & ~3) * (long long)sizeof(float) +
                        2 * (long long)sizeof(uint64_t);
    return (o + 127) / 128 * 128;
}

__device__ __forceinline__ void init_bars(uint64_t *bar, int n = 2) {
    if (threadIdx.x == 0) {
        for (int i = 0; i < n; i++) dd_mbar_init(&bar[i], 1);
        dd_fence_mbar_init();
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// Adjoint-type kernels (ProjTrans, BackProj, BackProjWeighted): pixel gathers.
// ---------------------------------------------------------------------------
constexpr int kLinesPerWarp = kTile / kWarps;   // fan beams: a thread's pixels

// Fan: the detector bin of axis position u, by the inverse of the fan's map
// (within one bin; fan_bin settles it on the exact boundaries).
__device__ __forceinline__ void det_index_fan(int geom, const dd_geom2d &g, const DdView2 &vw,
                                              float view, float u, int *kk) {
    const int D = g.num_det;
    float kf;
    if (geom == DD_GEOM_FLAT) {
        const float R = g.iso_source;
        const float vds = FMUL(FDIV(R, g.source_detector), g.det_size);
        const float vbs = FMUL(FDIV(R, g.source_detector), g.bin_shift);
        // virtual-detector coordinate of the ray source -> (u on the axis)
        const float t = vw.xb ? R * u * vw.c / (R + u * vw.s) : R * u * vw.s / (R - u * vw.c);
        const float q = (t - vbs) / vds;
        kf = vw.flip ? (float)D * 0.5f - q : q + (float)D * 0.5f;
    } else {
        // arc: angle of the ray through the axis point
        float ang = vw.xb ? atan2f(u - vw.srcx, vw.srcy) : 1.5707963267948966f - atanf((u - vw.srcy) / vw.srcx);
        const float base = view + g.bin_shift;
        ang += 3.14159265358979f * rintf((base - ang) * 0.3183098861837907f);
        const float q = (ang - base) / g.det_size;
        kf = vw.flip ? (float)D * 0.5f - q : q + (float)D * 0.5f;
    }
    int k = (int)floorf(kf);
    *kk = min(max(k, 0), D - 1);
}

// Detector-table entries per image staged in shared memory for one view
// (fan beams): the bins a 32x32 tile can touch.  Views whose range is wider
// gather from global memory instead.
constexpr int kStage = 256;

// Views in flight in the fan-beam adjoint: the copies of view v + 2 are issued
// while view v is computed (part of the map comes from HBM).
constexpr int kAdjBufs = 3;

static_assert((kAdjBufs * kMapBlkBytes + kAdjBufs * kBI * kStage * 8) % 16 == 0,
              "the fan adjoint's per-buffer copy descriptors must be 16-byte aligned");

// Shared-memory layout of the fan-beam adjoint (bytes): adjoint-map rows,
// detector table slices and per-line scales.
struct AdjSmem {
    int map, stage, krange, bar, total;
};

__host__ __device__ inline AdjSmem adj_smem() {
    AdjSmem s;
    int o = 0;
    s.map = o; o += kAdjBufs * kMapBlkBytes;
    s.stage = o; o += kAdjBufs * kBI * kStage * (int)sizeof(float2);
    s.krange = o; o += 4 * kAdjBufs * (int)sizeof(int);   // 16-byte aligned: read as int4
    s.bar = o; o += kAdjBufs * (int)sizeof(uint64_t);
    s.total = (o + 127) & ~127;
    return s;
}

// Detector bins [kmin, kmax] that pixels of the tile at (c0, r0) can reach at
// one view (fan beams): the walked pixel boundaries lie inside the tile's
// rectangle, whose central projection onto the axis spans the projections of
// its four corners.  Two bins of margin absorb rounding.
__device__ __forceinline__ void tile_bin_range(int geom, const dd_geom2d &g, const DdView2 &vw, float view, int c0,
                                               int r0, int *kmin, int *kmax) {
    const int W = g.width, H = g.height;
    const float xs[2] = {((float)c0 - 0.5f * W) * g.pix_x + g.pix_xshift,
                         ((float)min(c0 + kTile, W) - 0.5f * W) * g.pix_x + g.pix_xshift};
    const float ys[2] = {(0.5f * H - (float)r0) * g.pix_y + g.pix_yshift,
                         (0.5f * H - (float)min(r0 + kTile, H)) * g.pix_y + g.pix_yshift};
    int lo = g.num_det, hi = -1;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float px = xs[i & 1], py = ys[i >> 1];
        const float u = vw.xb ? dd_map2x(vw.srcx, vw.srcy, px, py) : dd_map2y(vw.srcx, vw.srcy, px, py);
        int k;
        det_index_fan(geom, g, vw, view, u, &k);
        lo = min(lo, k);
        hi = max(hi, k);
    }
    *kmin = max(lo - 2, 0);
    *kmax = min(hi + 2, g.num_det - 1);
}

// Detector-table position of axis value uu (fan beams): bin k with
// d_k <= uu < d_{k+1} (corrected against the exact table), clamped to the
// walked bins.  Returns k and d_k.
__device__ __forceinline__ int fan_bin(int geom, const dd_geom2d &g, const DdView2 &vw, float view,
                                       const float *__restrict__ dpv, float uu, int idet0, float *dk_out) {
    const int D = g.num_det;
    int k;
    det_index_fan(geom, g, vw, view, uu, &k);
    float dk = __ldg(dpv + k);
    if (k > 0 && uu < dk) {
        k--;
        dk = __ldg(dpv + k);
    } else if (k < D - 1 && uu >= __ldg(dpv + k + 1)) {
        k++;
        dk = __ldg(dpv + k);
    }
    if (k < idet0) {
        k = idet0;
        dk = __ldg(dpv + k);
    }
    *dk_out = dk;
    return k;
}

// One adjoint work item of one instance and a group of <= kBI of its images:
// fan beams, a 32x32 tile over all views; parallel beam, a walked line over
// the views that walk its axis.  Epilogue: out = value, or out = base + scale
// * value (base may alias out: in-place update).
struct AdjItem {
    int c0, r0, b0, nb, V, nl;   // parallel beam: c0 = line, r0 = 1 for rows, 0 for columns
    const DdView2 *views;
    const DdLine *lines, *dlines;   // parallel beam
    const unsigned char *amap;   // fan beams: adjoint-map blocks (plan)
    const int2 *trange;          // fan beams, per (view, tile): {first staged bin, bins | xb << 16} (plan)
    const int *axisv;            // view lists (plan)
    const float2 *dtab;          // detector tables of image 0 of the instance
    float *out;                  // image 0 of the instance
    const float *base;
    float scale;
};

// An adjoint tile or line is shared by a cluster of kAdjCluster CTAs, each
// taking a part of its views; the ranks' sums are added in rank order.
constexpr int kAdjCluster = 4;

// ---------------------------------------------------------------------------
// Fan-beam adjoint through the adjoint map, one 32 x 32 tile by a cluster of
// kAdjCluster CTAs.  Each CTA takes a part of the views that walk one axis and
// sums them on its own; the ranks' sums meet in shared memory at the end and
// are added in rank order, each rank writing a quarter of the tile.  So a
// tile's views are not one serial chain of copies, waits and barriers, and
// every view is walked along its own axis: a thread owns 4 consecutive pixels
// of one line (lane = line, warp = group of 4), whose 5 boundaries serve the
// 4 pixels.
//
// For every view the CTA copies by TMA the tile's map block -- the entries
// {bin, offset} of its lines' pixel boundaries and the lines' scales -- and
// the slice of every image's detector prefix table the tile can reach: pixel
// value += w (H(upper) - H(lower)), H(u) = G_k + (u - d_k) g_k.
//
// Bound by the map's stream from HBM for one slice (1.78 GB at 5.8 TB/s, 86 %
// of the copy rate) and by instruction issue (73 %) from 4 on.  512^2, 720
// views, 736 bins, 1 / 2 / 4 / 16 slices, by one CTA per tile with the pixels
// of views that walk rows on 4 lines a thread: 0.64 / 0.80 / 1.05 / 2.23 ms;
// here 0.35 / 0.41 / 0.53 / 1.87 ms (tables included).
// ---------------------------------------------------------------------------
static_assert(kTile % kAdjCluster == 0 && kTile / kAdjCluster == kWarps, "a rank writes one row per warp");

// Ranks that take the views walking rows (the others: columns), by their shares.
__device__ __forceinline__ int row_ranks(int nr, int nc) {
    if (nc == 0) return kAdjCluster;
    if (nr == 0) return 0;
    return min(max((int)((2ll * kAdjCluster * nr + nr + nc) / (2ll * (nr + nc))), 1), kAdjCluster - 1);
}

template <int GEOM, int OPK, int NB>   // OPK: 0 ProjTrans, 1 BackProj, 2 BackProjWeighted; NB: most images
__device__ bool adj_tile_map(const dd_geom2d &g, const AdjItem &it, unsigned char *smem, DdPhases &ph) {
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int rank = (int)cluster.block_rank();
    const AdjSmem SL = adj_smem();
    const int V = it.V;
    const int W = g.width, H = g.height, D = g.num_det;
    const int rsd = rs_entries(D);
    unsigned char *mapb = smem + SL.map;                           // [kAdjBufs] map blocks
    float2 *stage = reinterpret_cast<float2 *>(smem + SL.stage);   // [kAdjBufs][kBI][kStage]
    int *krange = reinterpret_cast<int *>(smem + SL.krange);       // per buffer: first bin, bins, first entry, view
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + SL.bar);
    __shared__ int abort_flag;
    const int c0 = it.c0, r0 = it.r0, b0 = it.b0, nb = it.nb;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float2 *__restrict__ dtab = it.dtab;
    if (tid == 0) abort_flag = 0;
    __syncthreads();

    // this rank's views: a part of one axis's list
    const int nr = it.axisv[0], nc = it.axisv[1], rk = row_ranks(nr, nc);
    const int xb = rank < rk;
    const int part = xb ? rank : rank - rk, parts = xb ? rk : kAdjCluster - rk, na = xb ? nr : nc;
    const int i0 = (int)((long long)na * part / parts), NV = (int)((long long)na * (part + 1) / parts) - i0;
    const int *__restrict__ vlist = it.axisv + 2 + (xb ? 0 : V) + i0;
    const int tile = (r0 / kTile) * tiles_x(&g) + c0 / kTile, ntiles = tiles_n(&g);
    const int elo = map_first(&g, xb, c0, r0);

    // thread 0 arms a buffer's barrier with the byte count of its next view
    // ({first staged bin, bins | xb << 16}), before any warp issues a copy into it
    auto arm = [&](int buf, int2 tr) {
        dd_mbar_expect_tx(&bar[buf], (uint32_t)(kMapBlkBytes + nb * (tr.y & 0xFFFF) * (int)sizeof(float2)));
    };
    // View v's copies, one per warp: warp 0 moves the tile's map block, warp
    // b + 1 (b < nb) the detector-table slice of image b.
    auto issue = [&](int v, int buf, int2 tr) {
        const int kn = tr.y & 0xFFFF;
        if (tid == 0) reinterpret_cast<int4 *>(krange)[buf] = make_int4(tr.x, kn, v, 0);
        if (lane == 0) {
            if (warp == 0)
                dd_bulk_g2s(mapb + (size_t)buf * kMapBlkBytes, it.amap + ((size_t)v * ntiles + tile) * kMapBlkBytes,
                            (uint32_t)kMapBlkBytes, &bar[buf]);
            else if (warp <= nb && kn > 0)
                dd_bulk_g2s(stage + ((size_t)buf * kBI + warp - 1) * kStage,
                            dtab + ((size_t)(b0 + warp - 1) * V + v) * rsd + tr.x, (uint32_t)(kn * sizeof(float2)),
                            &bar[buf]);
        }
    };

    float acc[kLinesPerWarp][NB];
#pragma unroll
    for (int q = 0; q < kLinesPerWarp; q++)
#pragma unroll
        for (int b = 0; b < NB; b++) acc[q][b] = 0.0f;

    // only the warps that issue a view's copies (warp 0: the map block, warps
    // 1 .. nb: the detector slices) follow the list ahead
    const bool issuing = warp <= nb;
    int vn = 0;                        // view i + 2 of the list, its range, and view i + 3
    int2 trn = make_int2(0, 0);
    int vnn = 0;
    {
        const int va = NV > 0 ? vlist[0] : 0, vb = NV > 1 ? vlist[1] : 0;
        const int2 ta = NV > 0 ? it.trange[(size_t)va * ntiles + tile] : make_int2(0, 0);
        const int2 tb = NV > 1 ? it.trange[(size_t)vb * ntiles + tile] : make_int2(0, 0);
        if (tid == 0) {
            if (NV > 0) arm(0, ta);
            if (NV > 1) arm(1, tb);
        }
        __syncthreads();
        if (NV > 0) issue(va, 0, ta);
        if (NV > 1) issue(vb, 1, tb);
        if (issuing) {
            if (NV > 2) {
                vn = vlist[2];
                trn = it.trange[(size_t)vn * ntiles + tile];
            }
            if (NV > 3) vnn = vlist[3];
        }
    }
    // this thread's 4 pixels: pixel q lies between entries E - q - 1 and E - q of its line
    const int rq0 = r0 + kLinesPerWarp * warp;
    const int E = xb ? kLinesPerWarp * (warp + 1) : H - rq0 - elo;
    const int nv = xb ? kLinesPerWarp : min(kLinesPerWarp, H - rq0);   // rows: absent pixels have no entries
    int vstop = NV;   // first view of the list not waited for (its copies may be in flight)
    int buf = 0, buf2 = 2 % kAdjBufs;   // buffers of views i and i + 2
    for (int i = 0; i < NV; i++, buf = (buf + 1 == kAdjBufs) ? 0 : buf + 1,
                                buf2 = (buf2 + 1 == kAdjBufs) ? 0 : buf2 + 1) {
        // the phase of view i - 1 on this barrier was waited for before the
        // previous barrier, so it can be armed for view i + 2 now
        if (tid == 0 && i + 2 < NV) arm(buf2, trn);
        if (!dd_mbar_wait(&bar[buf], ph.parity(buf))) abort_flag = 1;
        ph.flip(buf);
        // one barrier per view: past it every warp has finished view i - 1
        __syncthreads();
        if (abort_flag) {
            // view i's copies (not waited for) may still be in flight
            if (tid == 0) dd_mbar_drain(&bar[buf], ph.parity(buf) ^ 1u);
            vstop = i + 1;
            break;
        }
        // so the copies of view i + 2 go into the buffer of view i - 1
        if (issuing && i + 2 < NV) {
            issue(vn, buf2, trn);
            if (i + 3 < NV) {
                vn = vnn;
                trn = it.trange[(size_t)vn * ntiles + tile];
                if (i + 4 < NV) vnn = vlist[i + 4];
            }
        }
        const int4 kr = reinterpret_cast<const int4 *>(krange)[buf];   // one 16-byte load
        const int kb = kr.x, kn = kr.y, v = kr.z;
        const int2 *mp = reinterpret_cast<const int2 *>(mapb + (size_t)buf * kMapBlkBytes);
        const float *alb = reinterpret_cast<const float *>(mp + kTile * kMapE);   // line scales
        const float2 *sb = stage + (size_t)buf * kBI * kStage;
        if (nv > 0) {
            int2 m[kLinesPerWarp + 1];
            bool all_in = true;   // every used entry in the staged slice (the usual case)
#pragma unroll
            for (int e = 0; e <= kLinesPerWarp; e++) {
                m[e] = (e <= nv) ? mp[lane * kMapE + E - e] : make_int2(-1, 0);
                if (m[e].x >= 0 && (unsigned)(m[e].x - kb) >= (unsigned)kn) all_in = false;
            }
            float wq[kLinesPerWarp];
            if (OPK == 2) {
                const DdView2 *vw = it.views + v;   // the view's source and first pixel edge
                const float sx = vw->srcx, sy = vw->srcy, ax = vw->axis0;
#pragma unroll
                for (int q = 0; q < kLinesPerWarp; q++) {
                    const float pi = (float)(xb ? c0 + kLinesPerWarp * warp + 3 - q : H - 1 - (rq0 + q)) + 0.5f;
                    const float along = pix_centre(pi, xb ? g.pix_x : g.pix_y, ax);
                    const float across = xb ? pix_centre(0.5f * (float)H - (float)(r0 + lane) - 0.5f, g.pix_y, g.pix_yshift)
                                            : pix_centre((float)(c0 + lane) - 0.5f * (float)W + 0.5f, g.pix_x, g.pix_xshift);
                    wq[q] = alb[lane] * fan_fbp_weight<GEOM>(sx, sy, xb ? along : across, xb ? across : along, g.iso_source);
                }
            } else {
#pragma unroll
                for (int q = 0; q < kLinesPerWarp; q++) wq[q] = (OPK == 0) ? 1.0f : alb[lane];
            }
#pragma unroll
            for (int b = 0; b < NB; b++) {
                if (b >= nb) break;
                float h[kLinesPerWarp + 1];
                if (all_in) {
#pragma unroll
                    for (int e = 0; e <= kLinesPerWarp; e++) {
                        const float2 t = sb[b * kStage + max(m[e].x - kb, 0)];
                        h[e] = fmaf(__int_as_float(m[e].y), t.y, t.x);   // unused where m[e].x < 0
                    }
                } else {
                    const float2 *t = dtab + ((size_t)(b0 + b) * V + v) * rsd;   // per image
#pragma unroll
                    for (int e = 0; e <= kLinesPerWarp; e++) {
                        h[e] = 0.0f;
                        if (m[e].x >= 0) {
                            const bool in = (unsigned)(m[e].x - kb) < (unsigned)kn;
                            const float2 x = in ? sb[b * kStage + (m[e].x - kb)] : __ldg(t + m[e].x);
                            h[e] = fmaf(__int_as_float(m[e].y), x.y, x.x);
                        }
                    }
                }
#pragma unroll
                for (int q = 0; q < kLinesPerWarp; q++)
                    if (q < nv && m[q].x >= 0 && m[q + 1].x >= 0) acc[q][b] += wq[q] * (h[q] - h[q + 1]);
            }
        }
    }
    __syncthreads();   // the buffers are free: the last copies have been waited for ...
    if (abort_flag) {
        // ... or, after a timeout, are let land (those of view vstop, issued and not waited for)
        if (vstop < NV) {
            const int b = vstop % kAdjBufs;
            if (tid == 0) dd_mbar_drain(&bar[b], ph.parity(b));
            ph.flip(b);
        }
        __syncthreads();
    }
    // the ranks' sums, added in rank order
    float *sums = reinterpret_cast<float *>(mapb);   // [NB][kTile][kTile + 1]
#pragma unroll
    for (int b = 0; b < NB; b++)
#pragma unroll
        for (int q = 0; q < kLinesPerWarp; q++) {
            const int row = xb ? lane : kLinesPerWarp * warp + q, col = xb ? kLinesPerWarp * warp + 3 - q : lane;
            sums[(b * kTile + row) * (kTile + 1) + col] = acc[q][b];
        }
    cluster.sync();
    int ab = 0;
    for (int k = 0; k < kAdjCluster; k++) ab |= *cluster.map_shared_rank(&abort_flag, k);
    if (!ab) {
        const int row = rank * kWarps + warp, r = r0 + row, c = c0 + lane;
        if (r < H && c < W) {
#pragma unroll
            for (int b = 0; b < NB; b++) {
                if (b >= nb) break;
                const int at = (b * kTile + row) * (kTile + 1) + lane;
                float val = cluster.map_shared_rank(sums, 0)[at];
#pragma unroll
                for (int k = 1; k < kAdjCluster; k++) val += cluster.map_shared_rank(sums, k)[at];
                const size_t o = ((size_t)(b0 + b) * H + r) * W + c;
                it.out[o] = it.base ? fmaf(it.scale, val, it.base[o]) : val;
            }
        }
    }
    cluster.sync();   // no rank leaves (or reuses its buffers) before the others have read its sums
    return !ab;
}


// ---------------------------------------------------------------------------
// Parallel-beam adjoint, line-major.  The parallel beam's detector boundaries
// drift per walked line (ParaDisCPU2d.cpp:76, :100: the recurrence restarts
// at each line's first bin), so every (view, line, image) needs its own piece
// constants of the detector table.  A cluster takes one walked line and a
// group of images over all the views that walk its axis, each CTA a part of
// them: it builds the line's piece constants once per view and serves all the
// line's pixels from them, whose sums stay in shared memory.  The rows
// (x-branch views) are written by one launch and the columns added by a
// second.
//
// Where the lines fill the chip by themselves, one CTA takes a line: the same
// parts of its views in turn, added in the same order, so with equal bits, and
// without three more starts and a cluster's barriers.
//
// Bound by the chain of a view's steps (copy, piece constants, barrier, the
// locates) for a few slices: 256^2, 180 views, both launches, 1 / 4 slices 0.26 /
// 0.37 ms by one CTA a line, 0.17 / 0.23 ms by four; by the locates where the
// lines fill the chip by themselves: 16 slices of 512^2, 720 views, 9.3 -> 9.0.
// ---------------------------------------------------------------------------
struct ParaSmem {
    int rec, drec, tab, kt, acc, bar, total;
};
__host__ __device__ inline ParaSmem para_smem(int D, int npix, int nb) {
    ParaSmem s;
    int o = 0;
    s.rec = o; o += 2 * (int)sizeof(DdLine);
    s.drec = o; o += 2 * (int)sizeof(DdLine);
    s.tab = o; o += 2 * nb * rs_entries(D) * (int)sizeof(float2);
    s.kt = o; o += nb * 32 * (int)sizeof(float);
    s.acc = o; o += ((nb * npix + 3) & ~3) * (int)sizeof(float);
    s.bar = o; o += 2 * (int)sizeof(uint64_t);
    s.total = (o + 127) & ~127;
    return s;
}
// Pixels of a line that a thread adds to (its warp takes 31 of every 248).
__host__ __device__ inline int para_pixels(int npix) { return (npix + kWarps * kBinsPerWarp - 1) / (kWarps * kBinsPerWarp); }

// S: laid out for at least the item's detector, line and images.
// NQ > 0: one CTA, not a cluster, for lines of at most NQ pixels a thread.
template <int OPK, int NQ>   // OPK: 0 ProjTrans, 1 BackProj
__device__ bool adj_para_line(const dd_geom2d &g, const AdjItem &it, unsigned char *smem, const ParaSmem &S) {
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    constexpr bool ALONE = NQ > 0;
    const int rank = (int)cluster.block_rank();
    const int W = g.width, H = g.height, D = g.num_det, V = it.V;
    const int axis = it.r0, line = it.c0, b0 = it.b0, nb = it.nb;
    const int npix = axis ? W : H;
    const int na = it.axisv[axis ? 0 : 1];
    // part p of the axis's views ends before index part_end(p); a rank takes its own part, a single CTA all of them
    auto part_end = [&](int p) { return (int)((long long)na * (p + 1) / kAdjCluster); };
    const int v0 = ALONE ? 0 : part_end(rank - 1), nv = (ALONE ? na : part_end(rank)) - v0;
    const int *vlist = it.axisv + 2 + (axis ? 0 : V) + v0;
    const int rsd = rs_entries(D);
    DdLine *rec = reinterpret_cast<DdLine *>(smem + S.rec);
    DdLine *drec = reinterpret_cast<DdLine *>(smem + S.drec);
    float2 *tabs = reinterpret_cast<float2 *>(smem + S.tab);   // [2][nb][rsd]
    float *kt = reinterpret_cast<float *>(smem + S.kt);        // [nb][32]
    float *accs = reinterpret_cast<float *>(smem + S.acc);     // [nb][npix]
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + S.bar);
    __shared__ int abort_flag;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < nb * npix; i += kThreads) accs[i] = 0.0f;
    // a single CTA: the sums of the parts so far of the pixels that the thread adds to
    int part = 0;
    float sum[ALONE ? NQ : 1][kBI];
    auto close_part = [&]() {
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const int pi = (q * kWarps + warp) * kBinsPerWarp + lane - 1;
            const bool mine = lane > 0 && pi < npix;
#pragma unroll
            for (int b = 0; b < kBI; b++) {
                if (b >= nb || !mine) continue;
                float *x = accs + b * npix + pi;
                sum[q][b] = part == 0 ? *x : sum[q][b] + *x;
                *x = 0.0f;
            }
        }
        part++;
    };
    if (tid == 0) abort_flag = 0;
    init_bars(bar);   // synchronises the CTA
    DdPhases ph;

    const uint32_t rec_bytes = (uint32_t)sizeof(DdLine);
    const uint32_t tab_bytes = (uint32_t)(rsd * sizeof(float2));
    auto issue = [&](int idx, int buf) {
        const int v = vlist[idx];
        dd_mbar_expect_tx(&bar[buf], 2 * rec_bytes + nb * tab_bytes);
        dd_bulk_g2s(rec + buf, it.lines + (size_t)v * it.nl + line, rec_bytes, &bar[buf]);
        dd_bulk_g2s(drec + buf, it.dlines + (size_t)v * it.nl + line, rec_bytes, &bar[buf]);
        for (int b = 0; b < nb; b++)
            dd_bulk_g2s(tabs + ((size_t)buf * nb + b) * rsd, it.dtab + ((size_t)(b0 + b) * V + v) * rsd, tab_bytes,
                        &bar[buf]);
    };
    const int issuer = (kWarps - 1) * 32;
    if (tid == issuer && nv > 0) issue(0, 0);
    for (int idx = 0; idx < nv; idx++) {
        const int buf = idx & 1;
        if (!dd_mbar_wait(&bar[buf], ph.parity(buf))) abort_flag = 1;
        ph.flip(buf);
        // past this barrier every warp has finished view idx - 1, whose
        // buffer takes the copies of view idx + 1
        __syncthreads();
        if (abort_flag) {
            // view idx's copies (the wait gave up on them) may be in flight
            if (tid == issuer) dd_mbar_drain(&bar[buf], ph.parity(buf) ^ 1u);
            break;
        }
        if (tid == issuer && idx + 1 < nv) issue(idx + 1, buf ^ 1);
        if constexpr (ALONE)
            while (idx >= part_end(part)) close_part();
        const DdLine &L = rec[buf], &Ld = drec[buf];
        if (L.h.npiece == 0) continue;   // the same for the whole CTA
        const int npd = Ld.h.npiece;
        const float2 *tb = tabs + (size_t)buf * nb * rsd;
        for (int b = warp; b < nb; b += kWarps) kt[b * 32 + lane] = npd > 0 ? piece_K(Ld, tb + (size_t)b * rsd, lane) : 0.0f;
        __syncthreads();
        const int i0 = L.h.i0, nend = L.h.nend;
        const float bound0 = L.h.bound0;
        const float alpha = (OPK == 0) ? 1.0f : L.h.alpha;
        // a warp takes 32 consecutive pixel boundaries (lane l: the upper
        // boundary of pixel q0 + l - 1) and 31 pixels: each boundary is
        // located once and neighbours difference by one shuffle
        for (int q0 = warp * kBinsPerWarp; q0 < npix; q0 += kWarps * kBinsPerWarp) {   // warp-uniform
            const int bi = q0 + lane - 1;   // boundary index (upper boundary of pixel bi)
            float u = bound0;               // boundary i0 - 1 is the walk start; below it H is constant
            if (bi >= i0 && bi < nend) u = dd_boundary(&L, bi, L.p[0].Q + (float)(bi - L.p[0].gb) * L.p[0].dl);
            int pU = 0, jU = 0;
            float rU = 0.0f, dlU = 0.0f;
            if (npd > 0) {
                dd_locate(&Ld, fminf(fmaxf(u, bound0), Ld.h.endv), &pU, &jU, &rU);
                dlU = Ld.p[pU].dl;
            }
            const int pi = bi;   // the pixel this lane closes (lanes 1..31)
            const bool valid = lane > 0 && pi < npix && pi >= i0 && pi < nend;
#pragma unroll
            for (int b = 0; b < kBI; b++) {
                if (b >= nb) break;
                float hu = 0.0f;
                if (npd > 0) {
                    const float2 e = tb[(size_t)b * rsd + jU];
                    hu = fmaf(rU, e.y, fmaf(dlU, e.x, kt[b * 32 + pU]));
                }
                const float hl = __shfl_up_sync(0xffffffffu, hu, 1);
                if (valid) accs[b * npix + pi] += alpha * (hu - hl);
            }
        }
    }
    auto put = [&](int b, int pi, float val) {
        const int r = axis ? line : H - 1 - pi, c = axis ? pi : line;
        const size_t o = ((size_t)(b0 + b) * H + r) * W + c;
        if (axis) it.out[o] = it.base ? fmaf(it.scale, val, it.base[o]) : val;
        else it.out[o] = it.base ? fmaf(it.scale, val, it.out[o]) : it.out[o] + val;
    };
    if constexpr (ALONE) {
        __syncthreads();
        if (abort_flag) return false;
        while (part < kAdjCluster) close_part();
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const int pi = (q * kWarps + warp) * kBinsPerWarp + lane - 1;
            if (lane == 0 || pi >= npix) continue;
#pragma unroll
            for (int b = 0; b < kBI; b++)
                if (b < nb) put(b, pi, sum[q][b]);
        }
        return true;
    }
    cluster.sync();
    int ab = 0;
    for (int k = 0; k < kAdjCluster; k++) ab |= *cluster.map_shared_rank(&abort_flag, k);
    if (!ab) {
        const int n = nb * npix;
        for (int i = rank * kThreads + tid; i < n; i += kAdjCluster * kThreads) {
            const int b = i / npix, pi = i - b * npix;
            float val = cluster.map_shared_rank(accs, 0)[i];
#pragma unroll
            for (int k = 1; k < kAdjCluster; k++) val += cluster.map_shared_rank(accs, k)[i];
            put(b, pi, val);
        }
    }
    cluster.sync();   // no rank leaves before the others have read its sums
    return !ab;
}

// ---- host launchers shared by both translation units (dd2d.cu) -----------
struct ProfRec;
ProfRec *prof_begin(int kind, cudaStream_t st);
void prof_end(ProfRec *r, cudaStream_t st);
void count_launches(int n);
int plan(int scan, const dd_geom2d *g, const float *angles, int V, void *planp, size_t bytes,
         cudaStream_t st, bool with_map = true);
int validate(int scan, int op, const dd_geom2d *g, int B, int V);
int geom_of(int scan);
int launch_status();
int max_smem_optin();   // largest dynamic shared memory per CTA (opt-in) on this device
int sm_count();
// prefix tables of B sinograms of one geometry (adjoint)
int launch_det_tables(int geom, int op, const dd_geom2d *g, const char *planb, const float *in, int B,
                      int V, float2 *dtab, int *status, cudaStream_t st);   // clears *status

}  // namespace dd2
