// The arc fan's projection of one or two slices by prefix sums: with F the
// integral of a line's pixels, a bin's part of the line is F(upper boundary) -
// F(lower boundary), and on drift run p
//     F(u) = K_p + dl_p S_j + r x_j
// from the line's prefix table (S_j, x_j) and per-run constants.
//
// Why it stays beside the overlap forward (dd2d_fwd.cuh): for the values of the
// arc fan's A x that one or two slices have had, not for their accuracy.  A data-
// consistency block feeds A x to the ramp filter, and the gradient of its learned
// weight is a sum over the image that cancels: with overlaps it moved by up to
// 4.5e-4 (2 slices 3.1e-5; 2 x 512^2, 720 views, 768 cells, 10 inputs).  Against 64-bit sums over
// the same boundaries the overlaps are the nearer ones: A x 1.8e-7 against
// 6.7e-7 here, its filtered back-projection 1.5e-6 against 6.2e-6.  From three
// slices on they serve up to 8 at once (3 / 16 slices: 0.77 / 2.2 ms against
// 0.94 / 3.6 ms; 1 / 2 slices 0.64 / 0.72 against 0.69 / 0.80).
//
// A difference of two prefix sums rounds as the line's whole integral does: of
// N pixels, at c pixels a cell, over L lines, 2^-25 (N / c) sqrt(2 / L) of a bin's
// sum.  prefix_near keeps it below 1.4e-6; where cells are a small part of a pixel
// or lines few and long (1090 x 5 pixels, 1,984 cells: 1.4e-5 off the
// reference), overlaps serve one and two slices too.
//
// Bound by the shared-memory gathers and the search of the drift record per
// boundary, which one or two slices hardly share.
#pragma once

#include <cmath>

#include "dd2d_kernels.cuh"

namespace dd2 {

struct Loc {
    int p, j;
    float dl, r;
};

__device__ __forceinline__ Loc locate(const DdLine &L, float u) {
    Loc l;
    float rr;
    dd_locate(&L, u, &l.p, &l.j, &rr);
    l.r = rr;
    l.dl = L.p[l.p].dl;
    return l;
}

inline bool prefix_near(const dd_geom2d &g) {
    const double c = (double)g.det_size * g.iso_source / std::max(g.pix_x, g.pix_y), w = g.width, h = g.height;
    return std::max(w / std::sqrt(h), h / std::sqrt(w)) <= 32.0 * c;
}

// Detector passes of 8 warps x 31 bins, rounded up to the instantiated classes.
__host__ __device__ inline int prefix_passes(int D) {
    const int n = (D + kWarps * kBinsPerWarp - 1) / (kWarps * kBinsPerWarp);
    return n <= 1 ? 1 : n <= 2 ? 2 : n <= 3 ? 3 : n <= 4 ? 4 : 8;
}

struct PrefixSmem {
    int rec, tab, kt, dp, bar, total;
};
// The line tables' space also holds a CTA's sums for the cluster's combine.
__host__ __device__ inline PrefixSmem prefix_smem(int D, int rsmax, int bi) {
    PrefixSmem s;
    int o = 0;
    s.rec = o; o += 2 * (int)sizeof(DdLine);
    s.tab = o;
    {
        const int tabs = 2 * bi * rsmax * (int)sizeof(float2);
        const int red = prefix_passes(D) * bi * kThreads * (int)sizeof(float);
        o += tabs > red ? tabs : red;
    }
    s.kt = o; o += bi * 32 * (int)sizeof(float);   // K of the pixel pieces
    s.dp = o; o += ((D + 1 + 3) & ~3) * (int)sizeof(float);
    s.bar = o; o += 2 * (int)sizeof(uint64_t);
    s.total = (o + 127) & ~127;
    return s;
}

struct PrefixItem {
    int v, b0, nb, V, nl;
    const DdView2 *views;
    const float *dp, *bcoef;
    const DdLine *lines;
    const float2 *tabx, *taby;   // prefix tables of image 0
    float *out;                  // sinogram of image 0
    const float *sub;            // optional, same layout as out: out = A x - sub
};

// One view of a group of BI slices by a cluster of 2 CTAs: rank r walks lines
// r, r + 2, ..., with the line record and the line tables double-buffered in
// shared memory by bulk copies; rank 0 adds rank 1's sums.  Returns false if
// a bounded wait timed out (copies in flight have been drained).
template <int NPASS, int BI>
__device__ bool prefix_view(const dd_geom2d &g, const PrefixItem &it, unsigned char *smem, int rsmax,
                            DdPhases &ph) {
    constexpr int NW = kWarps, CL = 2;
    const int v = it.v, b0 = it.b0, nb = it.nb;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = (int)cooperative_groups::this_cluster().block_rank();
    const int D = g.num_det;
    const DdView2 vw = it.views[v];
    const int xb = vw.xb;
    const int nline = xb ? g.height : g.width;
    const int npix = xb ? g.width : g.height;
    const int rs = rs_entries(npix);
    const PrefixSmem L = prefix_smem(D, rsmax, BI);
    DdLine *rec = reinterpret_cast<DdLine *>(smem + L.rec);
    float2 *tab = reinterpret_cast<float2 *>(smem + L.tab);
    float *kt = reinterpret_cast<float *>(smem + L.kt);
    float *dps = reinterpret_cast<float *>(smem + L.dp);
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + L.bar);
    __shared__ int abort_flag;

    const float2 *tsrc = xb ? it.tabx : it.taby;
    const size_t img_stride = (size_t)nline * rs;          // float2 per image
    const uint32_t tab_bytes = (uint32_t)(rs * sizeof(float2));
    const uint32_t rec_bytes = (uint32_t)sizeof(DdLine);
    const uint32_t tx_bytes = nb * tab_bytes + rec_bytes;

    if (tid == 0) abort_flag = 0;
    for (int k = tid; k <= D; k += (NW * 32)) dps[k] = it.dp[(size_t)v * (D + 1) + k];
    __syncthreads();

    auto issue = [&](int line, int buf) {
        dd_mbar_expect_tx(&bar[buf], tx_bytes);
        dd_bulk_g2s(rec + buf, it.lines + (size_t)v * it.nl + line, rec_bytes, &bar[buf]);
        for (int b = 0; b < nb; b++)
            dd_bulk_g2s(tab + ((size_t)buf * BI + b) * rsmax,
                        tsrc + (size_t)(b0 + b) * img_stride + (size_t)line * rs, tab_bytes, &bar[buf]);
    };

    const int npass = (D + NW * kBinsPerWarp - 1) / (NW * kBinsPerWarp);
    constexpr int kMaxPass = NPASS;   // D <= NPASS * 248 detector bins
    float acc[kMaxPass][BI];
#pragma unroll
    for (int m = 0; m < kMaxPass; m++)
#pragma unroll
        for (int b = 0; b < BI; b++) acc[m][b] = 0.0f;

    // each pass's detector boundary is the same for all the lines of the view
    float ud[kMaxPass];
#pragma unroll
    for (int m = 0; m < kMaxPass; m++)
        ud[m] = (m < npass) ? dps[min(m * (NW * kBinsPerWarp) + warp * kBinsPerWarp + lane, D)] : 0.0f;
    // the last warp issues the copies: the first warps build the piece
    // constants right after the barrier, on every line's critical path
    const int issuer = (NW - 1) * 32;
    if (tid == issuer && rank < nline) issue(rank, 0);
    for (int line = rank, step = 0; line < nline; line += CL, step++) {
        const int buf = step & 1;
        if (!dd_mbar_wait(&bar[buf], ph.parity(buf))) abort_flag = 1;
        ph.flip(buf);
        // past this barrier every warp has finished line - 1, whose buffer
        // takes the copies of line + 1
        __syncthreads();
        if (abort_flag) {
            // this line's copies may still be in flight (the next line's are
            // issued only after this wait): let them land before returning
            if (tid == issuer) dd_mbar_drain(&bar[buf], ph.parity(buf) ^ 1u);
            break;
        }
        if (tid == issuer && line + CL < nline) issue(line + CL, buf ^ 1);
        const DdLine &R = rec[buf];
        const int np = R.h.npiece;
        if (np > 0) {
            const float2 *tb = tab + (size_t)buf * BI * rsmax;
            // warp b: image b's piece constants
            for (int b = warp; b < nb; b += NW) kt[b * 32 + lane] = piece_K(R, tb + (size_t)b * rsmax, lane);
            __syncthreads();
            const float bound0 = R.h.bound0, endv = R.h.endv;
            const int idet0 = R.h.idet0;
#pragma unroll
            for (int m = 0; m < kMaxPass; m++) {
                if (m >= npass) break;
                const int kb = m * (NW * kBinsPerWarp) + warp * kBinsPerWarp + lane;
                float u;
                if (kb <= idet0) {
                    u = bound0;   // lower boundary of bin idet0 is the walk start
                } else {
                    u = ud[m];
                }
                u = fminf(fmaxf(u, bound0), endv);
                // 32 boundaries clamped to the same end of the walk give 31
                // zero differences: the warp skips the bins this line misses
                if (__all_sync(0xffffffffu, u == bound0) || __all_sync(0xffffffffu, u == endv)) continue;
                const Loc lc = locate(R, u);
#pragma unroll
                for (int b = 0; b < BI; b++) {
                    if (b < nb) {
                        const float2 e = tb[(size_t)b * rsmax + lc.j];
                        const float f = fmaf(lc.r, e.y, fmaf(lc.dl, e.x, kt[b * 32 + lc.p]));
                        const float fn = __shfl_down_sync(0xffffffffu, f, 1);
                        if (lane < kBinsPerWarp) acc[m][b] += fn - f;
                    }
                }
            }
        }
    }
    // no copy is left in flight here: the next line's copies are issued only
    // after its predecessor's wait succeeded, and an abort drained its line's
    __syncthreads();   // the next item's first copies reuse the buffers
    // ranks > 0 leave their sums in the (idle) line-table space; rank 0
    // adds them in rank order, so the result does not depend on timing
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    float *red = reinterpret_cast<float *>(smem + L.tab);
    if (rank != 0 && !abort_flag) {
#pragma unroll
        for (int m = 0; m < kMaxPass; m++) {
            if (m >= npass) break;
#pragma unroll
            for (int b = 0; b < BI; b++) red[(m * BI + b) * (NW * 32) + tid] = acc[m][b];
        }
    }
    cluster.sync();
    int ab = 0;
    for (int r = 0; r < CL; r++) ab |= *cluster.map_shared_rank(&abort_flag, r);
    if (rank == 0 && !ab) {
        for (int r = 1; r < CL; r++) {
            const float *rr = cluster.map_shared_rank(red, r);
#pragma unroll
            for (int m = 0; m < kMaxPass; m++) {
                if (m >= npass) break;
#pragma unroll
                for (int b = 0; b < BI; b++) acc[m][b] += rr[(m * BI + b) * (NW * 32) + tid];
            }
        }
    }
    cluster.sync();   // no rank leaves (or reuses its buffers) before rank 0 has read them
    if (ab) return false;
    if (rank != 0) return true;
#pragma unroll
    for (int m = 0; m < kMaxPass; m++) {
        if (m >= npass) break;
        const int k = m * (NW * kBinsPerWarp) + warp * kBinsPerWarp + lane;
        if (lane < kBinsPerWarp && k < D) {
            const float beta = it.bcoef[(size_t)v * (D + 1) + k];
            const int ko = vw.flip ? D - 1 - k : k;
#pragma unroll
            for (int b = 0; b < BI; b++) {   // static indices keep acc in registers
                if (b >= nb) break;
                const size_t o = ((size_t)(b0 + b) * it.V + v) * D + ko;
                // rounded product, then rounded difference: bit-equal to a
                // separate projection followed by a subtraction (no FMA)
                float val = __fmul_rn(acc[m][b], beta);
                if (it.sub) val = __fsub_rn(val, it.sub[o]);
                it.out[o] = val;
            }
        }
    }
    return true;
}

// grid (views x cluster, 1): blockIdx.x = view * 2 + rank.
template <int NPASS, int BI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, (BI == 1 && NPASS <= 4) ? 8 : 0)
k_fwd_prefix(dd_geom2d g, int B, int V, int nl, const DdView2 *__restrict__ views,
             const float *__restrict__ dp, const float *__restrict__ bcoef, const DdLine *__restrict__ lines,
             const float2 *__restrict__ tabx, const float2 *__restrict__ taby, float *__restrict__ out,
             const float *__restrict__ sub, int *__restrict__ status) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int rsmax = rs_entries(g.width > g.height ? g.width : g.height);
    const PrefixSmem L = prefix_smem(g.num_det, rsmax, BI);
    init_bars(reinterpret_cast<uint64_t *>(smem + L.bar));
    DdPhases ph;
    PrefixItem it;
    it.v = blockIdx.x / 2;
    it.b0 = 0;
    it.nb = min(BI, B);
    it.V = V;
    it.nl = nl;
    it.views = views;
    it.dp = dp;
    it.bcoef = bcoef;
    it.lines = lines;
    it.tabx = tabx;
    it.taby = taby;
    it.out = out;
    it.sub = sub;
    if (!prefix_view<NPASS, BI>(g, it, smem, rsmax, ph) && threadIdx.x == 0) dd_report_timeout(status);
}

// ---------------------------------------------------------------------------
// Prefix tables of the images
// ---------------------------------------------------------------------------
// Row lines (x-branch): one warp per (image, row); S_j = sum_{i<j} x_i in
// double-float arithmetic, rounded once.  Entry n = (S_n, 0).
__global__ void k_tab_rows(const float *__restrict__ img, int B, int H, int W,
                           float2 *__restrict__ tab, int *__restrict__ clear) {
    if (blockIdx.x + threadIdx.x == 0) *clear = 0;   // the call's status word
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= B * H) return;
    const float *row = img + (size_t)warp * W;
    warp_prefix_table(W, tab + (size_t)warp * rs_entries(W), lane, [&](int j, float *x, float *w) {
        *x = row[j];
        *w = 1.0f;
    });
}

// Column lines (y-branch): line = image column, walked from the bottom row.
// A block takes 32 columns of one image (lanes: coalesced reads along a row)
// and splits the rows into kColChunks chunks (warps): each warp sums its
// chunk in double-float arithmetic, the chunk totals are added in order, and
// each warp then writes its rows' prefixes from its chunk's start -- 8 times
// the threads of one walk per column.
constexpr int kColChunks = 8;
__global__ void __launch_bounds__(32 * kColChunks)
k_tab_cols(const float *__restrict__ img, int B, int H, int W, float2 *__restrict__ tab) {
    const int c = threadIdx.x & 31, k = threadIdx.x >> 5;
    const int ncb = (W + 31) / 32;
    const int b = blockIdx.x / ncb, col = (blockIdx.x - b * ncb) * 32 + c;
    const int per = (H + kColChunks - 1) / kColChunks;
    const int i0 = min(H, k * per), i1 = min(H, i0 + per);
    const bool ok = b < B && col < W;
    const float *__restrict__ im = img + (size_t)b * H * W + col;
    __shared__ float tot_hi[kColChunks][32], tot_lo[kColChunks][32];
    DdF run = {0.0f, 0.0f};
    if (ok)
        for (int i = i0; i < i1; i++) run = df_add(run, DdF{__ldg(im + (size_t)(H - 1 - i) * W), 0.0f});
    tot_hi[k][c] = run.hi;
    tot_lo[k][c] = run.lo;
    __syncthreads();
    if (!ok) return;
    run = {0.0f, 0.0f};
    for (int q = 0; q < k; q++) run = df_add(run, DdF{tot_hi[q][c], tot_lo[q][c]});
    float2 *__restrict__ t = tab + ((size_t)b * W + col) * rs_entries(H);
    for (int i = i0; i < i1; i++) {
        const float x = __ldg(im + (size_t)(H - 1 - i) * W);
        t[i] = make_float2(run.hi, x);
        run = df_add(run, DdF{x, 0.0f});
    }
    if (i0 < H && i1 == H) t[H] = make_float2(run.hi, 0.0f);
}

}   // namespace dd2
