// The 2-D forward (Proj, BackProjTrans, BackProjTransWeighted: detector
// gathers) of one work item -- a view of one instance and up to NB of its
// slices -- shared by the single-geometry launch (dd2d.cu) and the persistent
// one over uneven instances (dd2d_batch.cu).
//
// A bin's part of a walked line is the sum of the line's pixels over the
// bin's interval on the projection axis.  With the line's drifted pixel
// boundaries at hand as a table, a thread finds the pixel its bin starts in
// by one multiply-add (the line is close to an arithmetic sequence; the
// estimate errs by at most one pixel, downwards), and walks the one to three pixels it
// meets: overlap, load, multiply-add per slice.  The overlaps are shared by
// the NB slices, whose pixels lie side by side.
//
// Producer warps evaluate the boundary tables from the lines' drift
// records (a few arithmetic runs per line) and start the bulk copies of the
// lines' pixels, several lines ahead of eight consumer warps; full and
// empty mbarriers order them, so there is no CTA barrier inside an item.
//
// Bound by instruction issue for few slices (about 1,700 a line: 36 per pass
// of 32 bins that meet it, a quarter for the tables) and by the shared-memory
// pipe for 8 (62 %, 1.4 wavefronts of each load being bank conflicts where
// bins step over pixels).  512^2, 720 views, 736 bins, tables included, 1 / 2
// / 4 / 16 slices: 0.70 / 0.87 / 1.02 / 3.6 ms by prefix sums (two table
// loads, a piece constant and a shuffle per boundary and slice, a search of
// the drift record per boundary, two CTA barriers a line) -> 0.66 / 0.72 /
// 0.79 / 2.18 ms.
#pragma once

#include <cmath>

#include "dd2d_kernels.cuh"

namespace dd2 {

// Eight consumer warps; producer warps (taking lines in turn) and lines between
// them and the slowest consumer, by slices per item.  512^2, 720 views, 736
// bins, ms for 1 / 2 / 4 / 16 slices: producers 4, 4, 4, 3 with stages 8, 6, 4,
// 3: 0.66 / 0.72 / 0.79 / 2.18; 2, 2, 2, 3 with 6, 4, 3, 4: 0.78 / 0.82 / 0.94
// / 3.07; 6, 6, 4, 3 with 8, 8, 6, 3: 0.68 / 0.76 / 0.86 / 2.18; 8, 5, 5, 4
// with 10, 8, 5, 4: 0.74 / 0.76 / 1.02 / 2.70.  Four consumer warps and twice
// the CTAs: 0.64 / 0.75 / 1.00, and 0.19 instead of 0.15 ms where views are
// few (parallel beam, 256^2, 180 views).
__host__ __device__ constexpr int pick4(int nb, int a, int b, int c, int d) { return nb == 1 ? a : nb == 2 ? b : nb == 4 ? c : d; }
__host__ __device__ constexpr int prods(int nb) { return pick4(nb, 4, 4, 4, 3); }
__host__ __device__ constexpr int stages(int nb) { return pick4(nb, 8, 6, 4, 3); }
constexpr int kCons = 8;
constexpr int kMaxRecs = 4;
constexpr int kMaxProd = 4, kMaxStages = 8;
constexpr int kBins = kCons * 32;   // bins of one pass of the consumers
__host__ __device__ constexpr int fwd_threads(int nb) { return (kCons + prods(nb)) * 32; }
static_assert(prods(1) <= stages(1) && prods(2) <= stages(2) && prods(4) <= stages(4) && prods(8) <= stages(8),
              "a producer must not wait for a stage two uses ahead of the consumers");

// Proj of a fan beam; the weighted DD back-projector's transpose of a fan beam
// (parts scaled per line and pixel); the parallel beam; the unweighted
// transpose of a fan beam (parts scaled per line); the weighted one without its
// table of weights.
enum { kFan = 0, kFanWeighted = 1, kPara = 2, kFanScaled = 3, kFanWeightedEach = 4 };
// Line records in flight per producer (the parallel beam's are twice as large).
__host__ __device__ constexpr int recs(int kind) { return kind == kPara ? 2 : kMaxRecs; }

// Passes over the detector, rounded up to the instantiated classes (the
// accumulators of a thread are NPASS x NB).
__host__ __device__ inline int pass_class(int D) {
    const int n = (D + kBins - 1) / kBins;
    return n <= 1 ? 1 : n <= 2 ? 2 : n <= 3 ? 3 : n <= 4 ? 4 : 8;
}

// Slices side by side: planes of P = min(NB, 4) slices per pixel, NB / P
// planes after one another, so that neighbouring lanes' 16-byte loads of
// neighbouring pixels hit distinct banks.
__host__ __device__ constexpr int plane_slices(int nb) { return nb < 4 ? nb : 4; }
// Pixels a line of a plane takes (a multiple of 16 bytes).
__host__ __device__ inline int plane_pitch(int n, int p) { return p == 1 ? (n + 3) & ~3 : p == 2 ? (n + 1) & ~1 : n; }
// Lanes a bin takes, as a power of two.  Bins of up to 4 pixels (parallel beam,
// whose passes cost more: 6) are one lane's; of wider ones a lane takes every
// 2nd, 4th ... 32nd pixel, three at a time: as many lanes as make passes x steps
// of three pixels fewest, within one pass, or two from 8 pixels on (fan beams).
// By the geometry alone: a slice's sums do not depend on how many are in the call.
//
// Flat fan, 1 / 8 slices, ms by prefix sums, a lane a bin, so.  512^2, 180 views:
// 16 cells 0.22, 0.34; 1.02, 1.52; 0.18, 0.27.  64 cells 0.22, 0.35; 0.36, 0.54;
// 0.19, 0.30.  128 cells 0.22, 0.36; 0.24, 0.37; 0.19, 0.32.  180 cells (3.4 pixels)
// 0.22, 0.37; 0.21, 0.33; two lanes 0.21, 0.37.  1000^2, 360 views: 16 cells 0.49,
// 1.98; 6.3, 12.5; 0.72, 1.50.  100 cells 0.49, 2.00; 1.41, 2.86; 0.96, 2.00.
// (Prefix sums ask for nothing per pixel but the tables' build: where views fill
// the chip they stay ahead for 1 to 4 slices of cells wider than 3 pixels -- 512^2,
// 720 views, 64 cells, 1 / 4 / 8 slices 0.45, 0.59, 1.07; so 0.55, 0.70, 0.90.)
inline int fwd_lanes(int geom, const dd_geom2d &g) {
    const bool para = geom == DD_GEOM_PARA;
    const double cell = para                   ? (double)g.det_size
                        : geom == DD_GEOM_FLAT ? (double)g.det_size * g.iso_source / g.source_detector
                                               : (double)g.det_size * g.iso_source;
    const double c = std::min(cell / std::min(g.pix_x, g.pix_y), 4096.0);   // pixels a bin, at the isocentre
    if (!(c > (para ? 6.0 : 4.0)) || g.num_det > kBins) return 0;
    double best = 1.0 + 0.7 * (c - 2.0);   // one lane: three pixels at once, the others in turn
    int sh = 0;
    for (int s = 1; s <= 5 && g.num_det << s <= 2 * kBins; s++) {
        const bool two = g.num_det << s > kBins;
        if (two && (para || !(c > 8.0))) break;
        const double cost = (two ? 2.0 : 1.0) * std::ceil((c + 1.0) / (3 << s));
        if (cost < best || (cost == best && two && g.num_det >= 64)) {   // (even: as measured)
            best = cost;
            sh = s;
        }
    }
    return sh;
}

// Bytes of a plane of P slices: its rows (h lines of w pixels) or columns.
__host__ __device__ inline size_t plane_bytes(int lines, int n, int p) {
    return sizeof(float) * (size_t)lines * plane_pitch(n, p) * p;
}

// Shared memory: a stage per line in flight {header, pixel boundaries, detector boundaries
// (parallel beam) or pixel weights (kFanWeighted), pixels}, line records, barriers.
struct FwdLay {
    int hdr, bnd, det, pix, red, rec, drec, bar, total;
    int bnd_b, det_b, pix_b;   // bytes of one stage
    int ks;                    // stages: stages(nb), or as many as fit
};
constexpr int kSmemMax = 227 * 1024;
// ... and to each of three CTAs on an SM, whose 228 KB also hold 1 KB per CTA
constexpr int kSmemThird = 228 * 1024 / 3 - 1024;
constexpr int kFwdStatic = 256;   // of either the kernels' static arrays take no more than this
// boundary e of a line sits at entry e + kB0 of its table
constexpr int kB0 = 4;
// lanes: the lanes that all bins take (D << fwd_lanes); ks: the stages.
__host__ __device__ inline FwdLay fwd_lay(int kind, int D, int lanes, int npix, int nb, int cl, int ks) {
    FwdLay s;
    const int p = plane_slices(nb);
    s.bnd_b = ((npix + kB0 + 8 + 3) & ~3) * (int)sizeof(float);
    const bool para = kind == kPara;
    s.det_b = para                   ? ((D + kB0 + 8 + 3) & ~3) * (int)sizeof(float)
              : kind == kFanWeighted ? ((npix + 3) & ~3) * (int)sizeof(float)
                                     : 0;
    s.pix_b = nb / p * plane_pitch(npix, p) * p * (int)sizeof(float);
    const int kP = prods(nb), red = pass_class(lanes) * nb * kCons * 32 * (int)sizeof(float);
    int o = 0;
    s.ks = ks;
    s.hdr = o; o += ks * 2 * (int)sizeof(float4);
    s.rec = o; o += kP * recs(kind) * (int)sizeof(DdLine);
    s.drec = o; o += para ? kP * recs(kind) * (int)sizeof(DdLine) : 0;
    s.bar = o; o += (2 * ks + recs(kind) * kP) * (int)sizeof(uint64_t);
    o = (o + 15) & ~15;
    s.bnd = o; o += ks * s.bnd_b;
    s.det = o; o += ks * s.det_b;
    // the sums of the even lines (cl = 1) or of the other CTA (cl = 2, after
    // the last line: in the pixels' space)
    s.pix = o; o += cl > 1 && red > ks * s.pix_b ? red : ks * s.pix_b;
    s.red = cl > 1 ? s.pix : o;
    if (cl == 1) o += red;
    s.total = (o + 127) & ~127;
    return s;
}
// With stages(nb) of them, or as many as fit; fewer for a third CTA on an SM,
// where the sums leave it registers and there is more than one a producer (24
// uneven parallel-beam instances of 1 to 3 slices: 10.3 ms with two CTAs, of 4
// records a producer and all stages; 7.9 ms with three).
inline FwdLay fwd_lay(int kind, int D, int lanes, int npix, int nb, int cl) {
    const int kP = prods(nb);
    auto of = [&](int ks) { return fwd_lay(kind, D, lanes, npix, nb, cl, ks); };
    int ks = stages(nb);
    while (ks > kP && of(ks).total + kFwdStatic > kSmemMax) ks--;
    if (pass_class(lanes) * nb <= 24)
        for (int k = ks; k > kP; k--)
            if (of(k).total + kFwdStatic <= kSmemThird) return of(k);
    return of(ks);
}

// Do NB slices side by side fit a CTA?
inline bool fwd_fits(int kind, int D, int lanes, int npix, int nb, int cl, int limit) {
    return fwd_lay(kind, D, lanes, npix, nb, cl).total + kFwdStatic <= limit;
}

struct FwdItem {
    int v, b0, nb, V, nl, sh;   // sh: log2 of the lanes a bin takes
    const DdView2 *views;
    const float *dp, *bcoef;
    const DdLine *lines, *dlines;
    const float *rows, *cols;      // the item's first plane of rows / columns
    size_t rplane, cplane;         // floats between planes
    float *out;                    // sinogram of image 0 of the instance
    const float *sub;              // optional: out = A x - sub
};

// What persists over a CTA's items (in static shared memory).
struct FwdState {
    int abort;
    int armed[kMaxStages];       // uses of each stage so far
    int nrec[kMaxProd][kMaxRecs];   // copies into each record buffer so far
};

// NB slices' values of one pixel, and sums of them.
template <int NB> struct Slices {
    static constexpr int N = NB / 2;
    unsigned long long v[N];     // packed pairs
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < N; i++) v[i] = 0ull;
    }
    __device__ __forceinline__ void add(float w, const float *pix, int plane) {
        unsigned long long w2;
        asm("mov.b64 %0, {%1, %1};" : "=l"(w2) : "f"(w));
        if constexpr (NB == 2) {
            const unsigned long long x = *reinterpret_cast<const unsigned long long *>(pix);
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v[0]) : "l"(w2), "l"(x));
        } else {
#pragma unroll
            for (int q = 0; q < NB / 4; q++) {
                const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(pix + (size_t)q * plane);
                asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v[2 * q]) : "l"(w2), "l"(x.x));
                asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v[2 * q + 1]) : "l"(w2), "l"(x.y));
            }
        }
    }
    __device__ __forceinline__ float get(int b) const {
        const unsigned long long p = v[b >> 1];
        return __uint_as_float((b & 1) ? (unsigned)(p >> 32) : (unsigned)p);
    }
    __device__ __forceinline__ void set(int b, float x) {
        const unsigned long long u = __float_as_uint(x);
        v[b >> 1] = (b & 1) ? ((v[b >> 1] & 0xFFFFFFFFull) | (u << 32)) : ((v[b >> 1] & ~0xFFFFFFFFull) | u);
    }
};
template <> struct Slices<1> {
    float v;
    __device__ __forceinline__ void clear() { v = 0.0f; }
    __device__ __forceinline__ void add(float w, const float *pix, int) { v = fmaf(w, *pix, v); }
    __device__ __forceinline__ float get(int) const { return v; }
    __device__ __forceinline__ void set(int, float x) { v = x; }
};

// Boundaries of a drift record into `t` (entry e + kB0), one warp: first eight
// at a time, each group from the run its first boundary lies in; then, one
// lane per run, the boundaries between a run's start and the end of the group
// it starts in.  Below the walk's start the table holds its value.  (A run's
// multiples of its increment are exact, so one FMA is the rounded sum.)
__device__ __forceinline__ void fill_boundaries(const DdLine &L, float *t, int lane) {
    const int i0 = L.h.i0, nend = L.h.nend, np = L.h.npiece;
    const DdPiece P0 = L.p[0];
#pragma unroll 2
    for (int e0 = (i0 & ~7) + 8 * lane; e0 < nend; e0 += 256) {
        const int p = dd_piece_of_index(&L, e0, FADD(P0.Q, FMUL((float)(e0 - P0.gb), P0.dl)));
        const DdPiece P = L.p[p];
        const float d = (float)(e0 - P.gb);
        float b[8];
#pragma unroll
        for (int i = 0; i < 8; i++) b[i] = fmaf(d + (float)i, P.dl, P.Q);
        float4 *o = reinterpret_cast<float4 *>(t + e0 + kB0);
        o[0] = make_float4(b[0], b[1], b[2], b[3]);
        o[1] = make_float4(b[4], b[5], b[6], b[7]);
    }
    __syncwarp();
    if (lane < np) {
        const DdPiece P = L.p[lane];
        const int f = lane > 0 ? L.p[lane - 1].gb + 1 : i0;
        const int end = min(P.gb, f | 7);
        for (int e = f; e <= end; e++) t[e + kB0] = fmaf((float)(e - P.gb), P.dl, P.Q);
    }
    __syncwarp();
    // the walk's start takes the place of the boundary below its first pixel
    if (lane == 0) t[i0 - 1 + kB0] = L.h.bound0;
}

// FBP weights of a line's pixels i0 .. nend - 1, one warp: once a pixel, where a
// weight per overlap is one per cell and pixel that meet.  Weighted transpose, 1
// / 4 / 8 / 16 slices, ms with the pixels weighed ahead of prefix tables / a
// weight per overlap / here: 512^2, 360 views, 736 bins 0.83, 1.29, 2.50, 4.69
// / 0.76, 0.88, 1.25, 2.26 / 0.45, 0.59, 0.80, 1.53; 300^2, 200 views, 1,200
// bins 0.44, 0.59, 1.12, 2.11 / 0.51, 0.75, 1.18, 2.24 / 0.27, 0.43, 0.69, 1.29.
// Lines of 900 to 1,000 pixels leave no room for 8 slices beside it: whole groups
// of 8 weigh each overlap there (kFanWeightedEach; 1000^2, 360 views, 900 bins, 8 /
// 16 slices 10.6, 18.5 / 3.3, 5.9, by groups of 4 with the table 3.9, 7.4).
template <int GEOM>
__device__ __forceinline__ void fill_weights(const dd_geom2d &g, const DdView2 &vw, int line, int i0, int nend, float *wt,
                                             int lane) {
    const int xb = vw.xb;
    const float sx = vw.srcx, sy = vw.srcy, axis0 = vw.axis0, pitch = xb ? g.pix_x : g.pix_y;
    const float lpos = xb ? pix_centre(0.5f * (float)g.height - (float)line - 0.5f, g.pix_y, g.pix_yshift)
                          : pix_centre((float)line - 0.5f * (float)g.width + 0.5f, g.pix_x, g.pix_xshift);
#pragma unroll 4
    for (int e = i0 + lane; e < nend; e += 32) {
        const float pc = pix_centre((float)e + 0.5f, pitch, axis0);
        wt[e] = fan_fbp_weight<GEOM>(sx, sy, xb ? pc : lpos, xb ? lpos : pc, g.iso_source);
    }
}

// Sets up a CTA's barriers and state (all threads; ends with a CTA barrier).
template <int KIND, int NB>
__device__ __forceinline__ void fwd_init(unsigned char *smem, const FwdLay &L, FwdState &S) {
    constexpr int kP = prods(NB), kRecs = recs(KIND);
    const int kS = L.ks;
    if (threadIdx.x == 0) {
        uint64_t *bar = reinterpret_cast<uint64_t *>(smem + L.bar);
        for (int i = 0; i < kS; i++) {
            dd_mbar_init(&bar[i], 2);             // full: the copy's byte count, and the tables
            dd_mbar_init(&bar[kS + i], kCons);    // empty
            S.armed[i] = 0;
        }
        for (int i = 0; i < kRecs * kP; i++) {
            dd_mbar_init(&bar[2 * kS + i], 1);    // records
            S.nrec[i / kRecs][i % kRecs] = 0;
        }
        S.abort = 0;
        dd_fence_mbar_init();
    }
    __syncthreads();
}

// One item.  `step` counts the CTA's lines so far, `nr` this producer warp's
// records (both kept by every warp, over the CTA's items).  Returns false if a
// bounded wait timed out (copies in flight have been drained).  The even and
// the odd lines are summed apart and then added: by a cluster of two CTAs
// side by side (rank 0 adds rank 1's sums through distributed shared memory),
// by a single CTA one after the other, with the same result bit for bit.
// WIDE: a bin may take more than one lane.
template <int KIND, int NPASS, int NB, bool WIDE>
__device__ bool fwd_item(const dd_geom2d &g, int geom, int op, const FwdItem &it, unsigned char *smem,
                         const FwdLay &L, FwdState &S, uint32_t &step, uint32_t &nr) {
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int CL = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    constexpr int P = plane_slices(NB), NPL = NB / P, kP = prods(NB), kRecs = recs(KIND);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int D = g.num_det, v = it.v;
    const int kS = L.ks;
    const DdView2 *vwp = it.views + v;
    const int xb = vwp->xb;
    const int nline = xb ? g.height : g.width;
    const int npix = xb ? g.width : g.height;
    const int pitch = plane_pitch(npix, P);
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + L.bar), *empty = full + kS;
    const int half = (nline + 1) / 2;   // even lines
    const int nstep = CL == 1 ? nline : rank == 0 ? half : nline - half;
    auto line_of = [&](int i) { return CL > 1 ? 2 * i + rank : i < half ? 2 * i : 2 * (i - half) + 1; };
    float *red = reinterpret_cast<float *>(smem + L.red);
    const int sh = WIDE ? it.sh : 0, lanes = 1 << sh, sub = lane & (lanes - 1);
    const int npass = ((D << sh) + kBins - 1) / kBins;
    Slices<NB> acc[NPASS];
#pragma unroll
    for (int m = 0; m < NPASS; m++) acc[m].clear();

    if (warp >= kCons) {
        const int p = warp - kCons;
        DdLine *rec = reinterpret_cast<DdLine *>(smem + L.rec) + kRecs * p;
        DdLine *drec = reinterpret_cast<DdLine *>(smem + L.drec) + kRecs * p;
        uint64_t *rbar = empty + kS + kRecs * p;
        const float *src = xb ? it.rows : it.cols;
        const size_t plane = xb ? it.rplane : it.cplane;
        const uint32_t row_b = (uint32_t)(pitch * P * (int)sizeof(float));
        auto issue = [&](int i, int buf) {   // the record of the item's step i (one lane)
            const size_t line = (size_t)v * it.nl + line_of(i);
            S.nrec[p][buf]++;
            dd_mbar_expect_tx(&rbar[buf], (uint32_t)sizeof(DdLine) * (KIND == kPara ? 2u : 1u));
            dd_bulk_g2s(rec + buf, it.lines + line, (uint32_t)sizeof(DdLine), &rbar[buf]);
            if (KIND == kPara) dd_bulk_g2s(drec + buf, it.dlines + line, (uint32_t)sizeof(DdLine), &rbar[buf]);
        };
        if (lane == 0) {
            for (int q = 0; q < kRecs; q++)
                if (p + q * kP < nstep) issue(p + q * kP, (nr + q) % kRecs);
        }
        __syncwarp();
        uint32_t st = (step + p) % (uint32_t)kS, use = (step + p) / (uint32_t)kS;
        for (int i = p; i < nstep; i += kP, nr++) {
            const int buf = (int)(nr % kRecs);
            bool ok = dd_mbar_wait(&rbar[buf], (nr / kRecs) & 1u);
            if (ok && use > 0) ok = dd_mbar_wait(&empty[st], (use - 1u) & 1u);
            if (!__all_sync(0xffffffffu, ok)) {
                S.abort = 1;
                break;
            }
            const DdLine &R = rec[buf];
            const int np = R.h.npiece, i0 = R.h.i0, nend = R.h.nend;
            if (lane == 0) {
                S.armed[st] = (int)use + 1;
                dd_mbar_expect_tx(&full[st], np > 0 ? NPL * row_b : 0u);
            }
            __syncwarp();
            if (np > 0) {
                if (lane < NPL)
                    dd_bulk_g2s(smem + L.pix + st * L.pix_b + lane * row_b,
                                src + (size_t)lane * plane + (size_t)line_of(i) * pitch * P, row_b, &full[st]);
                fill_boundaries(R, reinterpret_cast<float *>(smem + L.bnd + st * L.bnd_b), lane);
                if (KIND == kPara) fill_boundaries(drec[buf], reinterpret_cast<float *>(smem + L.det + st * L.det_b), lane);
                if (KIND == kFanWeighted) {
                    float *wt = reinterpret_cast<float *>(smem + L.det + st * L.det_b);
                    if (geom == DD_GEOM_ARC) fill_weights<DD_GEOM_ARC>(g, *vwp, line_of(i), i0, nend, wt, lane);
                    else fill_weights<DD_GEOM_FLAT>(g, *vwp, line_of(i), i0, nend, wt, lane);
                }
            }
            if (lane == 0) {
                // pixel of axis position u: inv u + off, the chord of the
                // boundaries less the most they deviate from it (half an ulp
                // per boundary) and the rounding: at most the pixel, and one
                // below it only within that distance of the pixel's start
                const DdPiece P0 = R.p[0];
                const float b0 = FADD(P0.Q, FMUL((float)(i0 - P0.gb), P0.dl));
                const float n = (float)(nend - 1 - i0), endv = R.h.endv;
                const float inv = nend - 1 > i0 ? __fdividef(n, endv - b0) : P0.invdl;
                const float slack = n * fmaxf(fabsf(b0), fabsf(endv)) * inv * 5.9604645e-8f + 1e-3f;
                const float off = fmaf(-b0, inv, (float)(i0 + 1)) - slack;
                float4 *h = reinterpret_cast<float4 *>(smem + L.hdr) + 2 * st;
                h[0] = make_float4(R.h.bound0, endv, inv, off);
                h[1] = make_float4(__int_as_float(i0), __int_as_float(np > 0 ? nend - i0 : 0),
                                   __int_as_float(R.h.idet0), op == DD_OP_PROJ ? 1.0f : R.h.alpha);
            }
            __syncwarp();   // the record has been read, the tables are written
            if (lane == 0) {
                dd_mbar_arrive(&full[st]);
                if (i + kRecs * kP < nstep) issue(i + kRecs * kP, buf);
            }
            if ((st += kP) >= (uint32_t)kS) {   // kP <= kS
                st -= kS;
                use++;
            }
        }
    } else {
        // fan beams: each pass's bin boundaries are the same for all lines
        float u0[NPASS], u1[NPASS];
#pragma unroll
        for (int m = 0; m < NPASS; m++) {
            const int k = (m * kBins + warp * 32 + lane) >> sh;
            u0[m] = 0.0f;
            u1[m] = -3.0e38f;   // past the detector: an empty interval
            if (KIND != kPara && k < D) {
                u0[m] = __ldg(it.dp + (size_t)v * (D + 1) + k);
                u1[m] = __ldg(it.dp + (size_t)v * (D + 1) + k + 1);
            }
        }
        uint32_t st = step % (uint32_t)kS, par = (step / (uint32_t)kS) & 1u;
        for (int i = 0; i < nstep; i++) {
            const bool ok = dd_mbar_wait(&full[st], par);
            if (!__all_sync(0xffffffffu, ok)) {
                S.abort = 1;
                break;
            }
            const float4 *h = reinterpret_cast<const float4 *>(smem + L.hdr) + 2 * st;
            const float4 h0 = h[0], h1 = h[1];
            const int n = __float_as_int(h1.y);
            if (n > 0) {
                const float bound0 = h0.x, endv = h0.y;
                const int idet0 = __float_as_int(h1.z);
                const int i0 = __float_as_int(h1.x), last = i0 + n - 1;
                const float *bt = reinterpret_cast<const float *>(smem + L.bnd + st * L.bnd_b) + kB0;
                float lpos = 0.0f;
                if (KIND == kFanWeightedEach) {
                    const int line = line_of(i);
                    lpos = xb ? pix_centre(0.5f * (float)g.height - (float)line - 0.5f, g.pix_y, g.pix_yshift)
                              : pix_centre((float)line - 0.5f * (float)g.width + 0.5f, g.pix_x, g.pix_xshift);
                }
                // the detector's boundaries, or the pixels' weights
                const float *dt = reinterpret_cast<const float *>(smem + L.det + st * L.det_b) + (KIND == kPara ? kB0 : 0);
                const float *pix = reinterpret_cast<const float *>(smem + L.pix + st * L.pix_b);
#pragma unroll
                for (int m = 0; m < NPASS; m++) {
                    if (m >= npass) break;
                    const int k = (m * kBins + warp * 32 + lane) >> sh;
                    // the bin's interval, clamped to the walk
                    float lo, hi;
                    if (KIND == kPara) {
                        // (the table starts just below bin idet0)
                        const int kc = min(max(k, idet0), D - 1);
                        lo = k <= idet0 ? bound0 : fmaxf(dt[kc - 1], bound0);
                        hi = k < idet0 || k >= D ? bound0 : fminf(dt[kc], endv);
                    } else {
                        lo = fmaxf(u0[m], bound0);
                        hi = fminf(u1[m], endv);
                    }
                    if (!__any_sync(0xffffffffu, lo < hi)) continue;   // 32 bins that miss the line
                    // the pixel the interval starts in, or the one below; an
                    // empty interval's parts are all empty
                    const int j = max(min((int)fmaf(lo, h0.z, h0.w), last), i0 - 1);
                    const float *b = bt + j;
                    auto add = [&](float w, int i) {   // a part of pixel j + i
                        if (!(w > 0.0f)) return;
                        if (KIND != kFan) w *= h1.w;
                        if (KIND == kFanWeighted) w *= dt[j + i];
                        if (KIND == kFanWeightedEach) {
                            const float pc = pix_centre((float)(j + i) + 0.5f, xb ? g.pix_x : g.pix_y, vwp->axis0);
                            const float cx = xb ? pc : lpos, cy = xb ? lpos : pc;
                            w *= geom == DD_GEOM_ARC
                                     ? fan_fbp_weight<DD_GEOM_ARC>(vwp->srcx, vwp->srcy, cx, cy, g.iso_source)
                                     : fan_fbp_weight<DD_GEOM_FLAT>(vwp->srcx, vwp->srcy, cx, cy, g.iso_source);
                        }
                        acc[m].add(w, pix + (j + i) * P, pitch * P);
                    };
                    if constexpr (!WIDE) {
                        // (past the last boundary, which bounds hi, the table may
                        // hold anything: what starts there is empty)
                        const float f0 = b[0], f1 = b[1], f2 = b[2];
                        const float g1 = fmaxf(f0, lo), g2 = fmaxf(f1, g1);
                        add(FSUB(fminf(f0, hi), lo), 0);
                        add(FSUB(fminf(f1, hi), g1), 1);
                        add(FSUB(fminf(f2, hi), g2), 2);
                        float from = fmaxf(f2, g2);
                        if (__any_sync(0xffffffffu, from < hi)) {   // bins of a few pixels more
                            for (int i = 3; from < hi && j + i <= last; i++) {
                                const float f = b[i];
                                add(FSUB(fminf(f, hi), from), i);
                                from = fmaxf(f, from);
                            }
                        }
                    } else {   // wide bins: a lane takes every lanes-th pixel, three at a time
                        int e = j + sub;
                        do {
#pragma unroll
                            for (int q = 0; q < 3; q++) {   // (entry last + 1, as above: empty)
                                const int i = min(e + q * lanes, last + 1);
                                add(FSUB(fminf(bt[i], hi), fmaxf(bt[i - 1], lo)), i - j);
                            }
                            e += 3 * lanes;
                        } while (e <= last && bt[e - 1] < hi);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) dd_mbar_arrive(&empty[st]);
            if (++st == (uint32_t)kS) {
                st = 0;
                par ^= 1u;
            }
            if (CL == 1 && i + 1 == half) {   // the even lines are done
#pragma unroll
                for (int m = 0; m < NPASS; m++) {
                    if (m >= npass) break;
#pragma unroll
                    for (int b = 0; b < NB; b++) red[(m * NB + b) * (kCons * 32) + tid] = acc[m].get(b);
                    acc[m].clear();
                }
            }
        }
    }
    step += (uint32_t)nstep;
    __syncthreads();
    bool ab = S.abort != 0;
    if (ab && tid == 0) {
        // let the copies in flight land: the last use of each barrier
        for (int i = 0; i < kS; i++)
            if (S.armed[i] > 0) dd_mbar_drain(&full[i], (uint32_t)(S.armed[i] - 1) & 1u);
        for (int p = 0; p < kP; p++)
            for (int b = 0; b < kRecs; b++)
                if (S.nrec[p][b] > 0) dd_mbar_drain(&empty[kS + kRecs * p + b], (uint32_t)(S.nrec[p][b] - 1) & 1u);
    }
    auto add = [&](const float *r) {   // (sums of the even lines) + (sums of the odd ones)
#pragma unroll
        for (int m = 0; m < NPASS; m++) {
            if (m >= npass) break;
#pragma unroll
            for (int b = 0; b < NB; b++) acc[m].set(b, acc[m].get(b) + r[(m * NB + b) * (kCons * 32) + tid]);
        }
    };
    if (CL > 1) {
        if (rank != 0 && !ab && warp < kCons) {
#pragma unroll
            for (int m = 0; m < NPASS; m++) {
                if (m >= npass) break;
#pragma unroll
                for (int b = 0; b < NB; b++) red[(m * NB + b) * (kCons * 32) + tid] = acc[m].get(b);
            }
            dd_fence_async();   // the next item's copies land where these sums lie
        }
        cluster.sync();
        for (int r = 0; r < CL; r++) ab = ab || *cluster.map_shared_rank(&S.abort, r) != 0;
        if (rank == 0 && !ab && warp < kCons) add(cluster.map_shared_rank(red, 1));
        cluster.sync();   // no rank leaves (or reuses its buffers) before rank 0 has read them
    } else if (!ab && warp < kCons) {
        add(red);
    }
    if (ab) return false;
    if (rank != 0 || warp >= kCons) return true;
    if constexpr (WIDE) {   // a bin's lanes, each other's sums by halves: the same order for any group of slices
#pragma unroll
        for (int m = 0; m < NPASS; m++) {
            if (m >= npass) break;
#pragma unroll
            for (int b = 0; b < NB; b++) {
                float x = acc[m].get(b);
                for (int o = 1; o < lanes; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                acc[m].set(b, x);
            }
        }
    }
    const float para_beta = xb ? FDIV(g.pix_y, g.det_size) : FDIV(g.pix_x, g.det_size);
#pragma unroll
    for (int m = 0; m < NPASS; m++) {
        if (m >= npass) break;
        const int k = (m * kBins + warp * 32 + lane) >> sh;
        if (k >= D || sub != 0) continue;
        float beta = 1.0f;
        if (op == DD_OP_PROJ) beta = (KIND == kPara) ? para_beta : it.bcoef[(size_t)v * (D + 1) + k];
        const int ko = vwp->flip ? D - 1 - k : k;
#pragma unroll
        for (int b = 0; b < NB; b++) {
            if (b >= it.nb) break;
            const size_t o = ((size_t)(it.b0 + b) * it.V + v) * D + ko;
            // rounded product, then rounded difference: bit-equal to a
            // separate projection followed by a subtraction (no FMA)
            float val = __fmul_rn(acc[m].get(b), beta);
            if (it.sub) val = __fsub_rn(val, it.sub[o]);
            it.out[o] = val;
        }
    }
    return true;
}

// A 32 x 32 tile of one plane: slices [b0, b0 + P) (zero from nb on) of an
// image stack into the plane's rows [y][x] and columns [x][H-1-y], the slices
// of a pixel side by side.  One CTA of 256 threads; t: 32 x 33 pixels.
template <int P>
__device__ __forceinline__ void plane_tile(const float *__restrict__ img, int nb, int W, int H, int x0, int y0,
                                           float *__restrict__ rows, float *__restrict__ cols, float (*t)[33 * P]) {
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int wr = plane_pitch(W, P), wc = plane_pitch(H, P);
    const size_t one = (size_t)W * H;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int y = y0 + ty + 8 * i, x = x0 + tx;
        if (y < H && x < W) {
            const float *s = img + (size_t)y * W + x;
            float *r = rows + ((size_t)y * wr + x) * P;
#pragma unroll
            for (int b = 0; b < P; b++) {
                const float val = b < nb ? s[b * one] : 0.0f;
                t[ty + 8 * i][tx * P + b] = val;
                r[b] = val;
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int x = x0 + ty + 8 * i, y = y0 + tx;
        if (x < W && y < H) {
            float *c = cols + ((size_t)x * wc + (H - 1 - y)) * P;
#pragma unroll
            for (int b = 0; b < P; b++) c[b] = t[tx][(ty + 8 * i) * P + b];
        }
    }
}

}   // namespace dd2
