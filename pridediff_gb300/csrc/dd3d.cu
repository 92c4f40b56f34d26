// 3-D DD projector (cone-flat, cone-arc, spiral): plan kernels, the
// forward-type kernel (detector gathers) and the adjoint-type kernel (voxel
// gathers), and the C ABI of include/pridediff_dd.h for the 18 3-D
// radontorch operators (RadonTorch.cpp:1395-1414).
//
// Forward-type operators (Proj, BackProjTrans, BackProjTransWeighted): one
// thread per (view, column, up to 8 detector rows, 2 or 1 volumes) loops over
// the walked image lines.  For each line the overlap segments of the columns
// with the drifted pixel boundaries (dd3_colwalk_*) are summed once per slice,
// and every row then merges its interval with the slices.  Volumes are read
// from copies in which the pixels of a walked line are contiguous in both
// branches.
//
// Adjoint-type operators (ProjTrans, BackProj, BackProjWeighted): one thread
// per (x, y) voxel column, 16 or 8 slices and 2 or 1 volumes loops over the
// views; for each view it enumerates the segments of its pixel with the
// detector columns and merges the column's rows with its slices, reading a
// sinogram pre-multiplied by the per-bin scale.  Views whose detector cannot
// see the CTA's slices (most views of a spiral scan) are left out of its list.
//
// Both directions use the same segment widths and z-walk widths, so they are
// exact transposes of each other; no atomics, deterministic results.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/pridediff_dd.h"
#include "dd_geom3d.cuh"
#include "dd_tma.cuh"
#include "dd_trace.h"

namespace dd2 {   // launch accounting and profiling (dd2d.cu)
struct ProfRec;
ProfRec *prof_begin(int kind, cudaStream_t st);
void prof_end(ProfRec *r, cudaStream_t st);
void count_launches(int n);
}   // namespace dd2

namespace dd3 {

constexpr int kThreads = 256;
constexpr int kNB = 2;     // volumes per thread (an odd last volume runs on its own)
constexpr int kTile = 16;  // adjoint: 16 x 16 voxel columns per CTA
constexpr int kZS = 8;     // adjoint: slices of a slab (a thread takes one slab or two)

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// ---------------------------------------------------------------------------
// Layouts
// ---------------------------------------------------------------------------
// Per-view tables are padded to 16-byte rows so that one view's row can be
// moved by a single bulk copy: dp (C+1 column boundaries), mag (C column
// magnifications), rowz (R x {row0z, row1z}, closed by a row at infinity).
struct PlanLayout {
    size_t views, dp, mag, rowz, linez, lines, slabv, total;
    int nl, nch, sdp, smag, srz, nslab;
};

__host__ __device__ inline int pad4(int n) { return (n + 3) & ~3; }

inline PlanLayout plan_layout(const dd_geom3d *g, int V) {
    PlanLayout L;
    const int C = g->num_col, R = g->num_row;
    L.nl = g->height > g->width ? g->height : g->width;
    L.nch = (C + DD3_CHUNK - 1) / DD3_CHUNK;
    L.sdp = pad4(C + 1);
    L.smag = pad4(C);
    L.srz = pad4(2 * R + 2);
    size_t o = 0;
    L.views = o; o = align_up(o + sizeof(DdView3) * (size_t)V, 256);
    L.dp = o; o = align_up(o + sizeof(float) * (size_t)V * L.sdp, 256);
    L.mag = o; o = align_up(o + sizeof(float) * (size_t)V * L.smag, 256);
    L.rowz = o; o = align_up(o + sizeof(float) * (size_t)V * L.srz, 256);
    L.linez = o; o = align_up(o + sizeof(float4) * (size_t)V * L.nl, 256);
    // line records [view][walk block][line]: a tile's 16 lines of one block are contiguous
    L.lines = o; o = align_up(o + sizeof(DdLine) * (size_t)V * L.nl * L.nch, 256);
    L.nslab = (g->depth + kZS - 1) / kZS;   // the adjoint's slabs of kZS slices
    L.slabv = o; o = align_up(o + sizeof(int2) * (size_t)L.nslab, 256);
    L.total = o;
    return L;
}

struct ApplyLayout {
    size_t volx, volt, ss, status, total;
};

inline bool op_is_forward(int op) { return op == DD_OP_PROJ || op == DD_OP_BPROJ_T || op == DD_OP_BPROJ_TW; }
inline int op_family(int op) {
    return (op == DD_OP_PROJ || op == DD_OP_PROJ_T) ? 0 : (op == DD_OP_BPROJ_W || op == DD_OP_BPROJ_TW) ? 2 : 1;
}

// fwd / adj select which scratch areas are needed (both for the DC step)
inline ApplyLayout apply_layout(bool fwd, bool adj, const dd_geom3d *g, int B, int V) {
    ApplyLayout L;
    size_t o = 0;
    L.volx = L.volt = L.ss = 0;
    if (fwd) {   // the volumes' rows and columns, padded to 16 bytes (k_lines_of3)
        L.volx = o; o = align_up(o + sizeof(float) * (size_t)B * g->depth * g->height * pad4(g->width), 256);
        L.volt = o; o = align_up(o + sizeof(float) * (size_t)B * g->depth * g->width * pad4(g->height), 256);
    }
    if (adj) { L.ss = o; o = align_up(o + sizeof(float) * (size_t)B * V * g->num_row * g->num_col, 256); }
    L.status = o; o = align_up(o + 256, 256);
    L.total = o;
    return L;
}

// A caller's workspace from its first 16-byte boundary on (tensor maps and the
// paired volumes' 8-byte loads need it).  The 256 bytes of the status words,
// which close every layout, leave room for the shift.
inline char *ws_base(const void *ws) { return (char *)(((uintptr_t)ws + 15) & ~(uintptr_t)15); }

// ---------------------------------------------------------------------------
// Plan kernels
// ---------------------------------------------------------------------------
// One CTA per view: scalars, column boundaries, column magnifications, row
// table, and the ranges used by the adjoint's candidate searches.
template <int GEOM>
__global__ void __launch_bounds__(kThreads) k_views3(dd_geom3d g, const float *__restrict__ angles,
                                                     const float *__restrict__ sp, int V, char *plan,
                                                     PlanLayout P) {
    const int v = blockIdx.x, tid = threadIdx.x;
    const int C = g.num_col, R = g.num_row;
    __shared__ DdView3 sw;
    __shared__ float red[2][kThreads / 32];
    if (tid == 0) {
        float sp4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (GEOM == DD_GEOM3_SPIRAL)
            for (int i = 0; i < 4; i++) sp4[i] = sp[(size_t)i * V + v];
        dd3_view_scalars(GEOM, &g, angles[v], sp4, &sw);
    }
    __syncthreads();
    const DdView3 w = sw;
    float *dp = reinterpret_cast<float *>(plan + P.dp) + (size_t)v * P.sdp;
    float *mag = reinterpret_cast<float *>(plan + P.mag) + (size_t)v * P.smag;
    float *rz = reinterpret_cast<float *>(plan + P.rowz) + (size_t)v * P.srz;
    for (int k = tid; k <= C; k += kThreads) dp[k] = dd3_col_boundary(GEOM, &g, &w, k);
    float mn = 3.0e38f, mx = -3.0e38f;
    for (int k = tid; k < C; k += kThreads) {
        const float m = dd3_col_mag(GEOM, &g, &w, k);
        mag[k] = m;
        mn = fminf(mn, m);
        mx = fmaxf(mx, m);
    }
    for (int r = tid; r < R; r += kThreads) dd3_row_z(GEOM, &g, &w, r, &rz[2 * r], &rz[2 * r + 1]);
    if (tid < 2) rz[2 * R + tid] = __int_as_float(0x7f800000);   // +inf: ends the adjoint's row walks
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((tid & 31) == 0) {
        red[0][tid >> 5] = mn;
        red[1][tid >> 5] = mx;
    }
    __syncthreads();
    if (tid == 0) {
        DdView3 out = w;
        out.magmin = red[0][0];
        out.magmax = red[1][0];
        for (int i = 1; i < kThreads / 32; i++) {
            out.magmin = fminf(out.magmin, red[0][i]);
            out.magmax = fmaxf(out.magmax, red[1][i]);
        }
        float a0, a1, b0, b1;
        dd3_row_z(GEOM, &g, &w, 0, &a0, &a1);
        dd3_row_z(GEOM, &g, &w, R - 1, &b0, &b1);
        out.rzA = a0;
        out.rzB = (R > 1) ? (b0 - a0) / (float)(R - 1) : a1 - a0;
        out.rzI = 1.0f / out.rzB;
        reinterpret_cast<DdView3 *>(plan + P.views)[v] = out;
    }
}

// One thread per (view, line, walk block): walk start and drift pieces.
template <int GEOM>
__global__ void __launch_bounds__(128) k_lines3(dd_geom3d g, char *plan, PlanLayout P) {
    const int v = blockIdx.y;
    const int idx = blockIdx.x * 128 + threadIdx.x;
    const int line = idx / P.nch, cc = idx - line * P.nch;
    const DdView3 *views = reinterpret_cast<const DdView3 *>(plan + P.views);
    const int xb = views[v].xb;
    const int nline = xb ? g.height : g.width;
    if (line >= nline) return;
    const DdView3 w = views[v];
    const float *dp = reinterpret_cast<const float *>(plan + P.dp) + (size_t)v * P.sdp;
    DdLine *L = reinterpret_cast<DdLine *>(plan + P.lines) + ((size_t)v * P.nch + cc) * P.nl + line;
    float lz[4];
    dd3_line_setup(GEOM, &g, &w, dp, line, cc, lz, L);
    if (cc == 0)
        reinterpret_cast<float4 *>(plan + P.linez)[(size_t)v * P.nl + line] = make_float4(lz[0], lz[1], lz[2], lz[3]);
}

// One volume's value, or two volumes' side by side: the adjoint's gathers move
// both with one 8-byte load.
template <int NB> struct Vox;
template <> struct Vox<1> {
    using T = float;
    static __device__ __forceinline__ T zero() { return 0.0f; }
    static __device__ __forceinline__ T fma(float w, T x, T a) { return fmaf(w, x, a); }
    using K = float;   // a coefficient used for all the volumes of several loads
    static __device__ __forceinline__ K coef(float w) { return w; }
    static __device__ __forceinline__ T kmul(K w, T x) { return FMUL(w, x); }
    static __device__ __forceinline__ T kfma(K w, T x, T a) { return fmaf(w, x, a); }
    static __device__ __forceinline__ float get(T x, int) { return x; }
};
template <> struct Vox<2> {
    using T = float2;
    static __device__ __forceinline__ T zero() { return make_float2(0.0f, 0.0f); }
    static __device__ __forceinline__ T fma(float w, T x, T a) { return make_float2(fmaf(w, x.x, a.x), fmaf(w, x.y, a.y)); }
    // two products at once (the packed FP32 instructions; each rounds as the scalar one)
    using K = unsigned long long;
    static __device__ __forceinline__ K coef(float w) {
        K k;
        asm("mov.b64 %0, {%1, %1};" : "=l"(k) : "f"(w));
        return k;
    }
    static __device__ __forceinline__ T kmul(K w, T x) {
        asm("{\n .reg .b64 t;\n mov.b64 t, {%0, %1};\n mul.rn.f32x2 t, %2, t;\n mov.b64 {%0, %1}, t;\n}"
            : "+f"(x.x), "+f"(x.y) : "l"(w));
        return x;
    }
    static __device__ __forceinline__ T kfma(K w, T x, T a) {
        asm("{\n .reg .b64 t, u;\n mov.b64 t, {%0, %1};\n mov.b64 u, {%3, %4};\n fma.rn.f32x2 t, %2, u, t;\n"
            " mov.b64 {%0, %1}, t;\n}"
            : "+f"(a.x), "+f"(a.y) : "l"(w), "f"(x.x), "f"(x.y));
        return a;
    }
    static __device__ __forceinline__ float get(T x, int b) { return b ? x.y : x.x; }
};

// The walked lines of either kind, each line's pixels contiguous, the volumes
// of a group of kNB next to each other (an odd last volume forms a group of
// its own), lines padded to a multiple of 4 pixels:
//   vx[s][y][x][b] = vol[b][s][y][x],  vt[s][x][H-1-y][b] = vol[b][s][y][x].
template <int NB>
__global__ void __launch_bounds__(256) k_lines_of3(const float *__restrict__ in, float *__restrict__ vx,
                                                   float *__restrict__ vt, int W, int H, int Dp, int ngroups,
                                                   int *__restrict__ clear) {
    if (clear && threadIdx.x == 0 && blockIdx.x + blockIdx.y + blockIdx.z == 0) *clear = 0;   // the call's status word
    using T = typename Vox<NB>::T;
    __shared__ T t[32][33];
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int Wp = pad4(W), Hp = pad4(H);
    const size_t vox = (size_t)W * H * Dp;
    for (int pl = blockIdx.z; pl < Dp * ngroups; pl += gridDim.z) {
        const int gr = pl / Dp, s = pl - gr * Dp;
        const float *__restrict__ src = in + (size_t)gr * NB * vox + (size_t)s * H * W;
        T *__restrict__ px = reinterpret_cast<T *>(vx) + ((size_t)gr * Dp + s) * H * Wp;
        T *__restrict__ pt = reinterpret_cast<T *>(vt) + ((size_t)gr * Dp + s) * W * Hp;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int y = y0 + ty + 8 * i, x = x0 + tx;
            if (y < H && x < W) {
                const size_t o = (size_t)y * W + x;
                T val;
                if constexpr (NB == 2) val = make_float2(src[o], src[vox + o]);
                else val = src[o];
                t[ty + 8 * i][tx] = val;
                px[(size_t)y * Wp + x] = val;
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int x = x0 + ty + 8 * i, y = y0 + tx;
            if (x < W && y < H) pt[(size_t)x * Hp + (H - 1 - y)] = t[tx][ty + 8 * i];
        }
        __syncthreads();
    }
}

// ss[v][r][k][b] = in[b][v][r][k'] * scale(v, r, k) with k the sorted column:
// the adjoint gathers pre-scaled bins (ConeFlatDisCUDA3d.cu:400-404), the
// volumes of a group of kNB next to each other (an odd last volume forms a
// group of its own).
template <int GEOM, int FAMILY>
__global__ void __launch_bounds__(128) k_sino3(dd_geom3d g, const char *__restrict__ plan, PlanLayout P,
                                               const float *__restrict__ in, float *__restrict__ ss, int B, int V,
                                               int *__restrict__ clear) {
    if (threadIdx.x + blockIdx.x + blockIdx.y + blockIdx.z == 0) *clear = 0;   // the call's status word
    const int C = g.num_col, R = g.num_row;
    const int k = blockIdx.x * 128 + threadIdx.x, r = blockIdx.y, v = blockIdx.z;
    if (k >= C) return;
    const DdView3 &w = reinterpret_cast<const DdView3 *>(plan + P.views)[v];
    float scale = w.bp_scale;
    if (FAMILY == 0) {
        const float *dp = reinterpret_cast<const float *>(plan + P.dp) + (size_t)v * P.sdp;
        const float *rz = reinterpret_cast<const float *>(plan + P.rowz) + (size_t)v * P.srz;
        const float mag = reinterpret_cast<const float *>(plan + P.mag)[(size_t)v * P.smag + k];
        float rp0, rp1;
        dd3_rp(GEOM, &w, mag, rz[2 * r], rz[2 * r + 1], &rp0, &rp1);
        scale = dd3_proj_scale(&g, &w, dp[k], dp[k + 1], rp0, rp1);
    }
    const int ko = w.flip ? C - 1 - k : k;
    const size_t per = (size_t)V * R * C;
    const size_t row = ((size_t)v * R + r) * C;
    int b = 0;
    for (; b + 1 < B; b += 2)
        reinterpret_cast<float2 *>(ss + b * per)[row + k] =
            make_float2(FMUL(in[b * per + row + ko], scale), FMUL(in[(b + 1) * per + row + ko], scale));
    if (b < B) ss[b * per + row + k] = FMUL(in[b * per + row + ko], scale);
}

// ---------------------------------------------------------------------------
// Forward-type kernel: detector gathers
// ---------------------------------------------------------------------------
constexpr int kFC = 32;      // detector columns per CTA (the lanes of a warp)
constexpr int kCons3 = 8;    // consumer warps
// Producer warps (taking steps in turn), stages between them and the slowest
// consumer, and CTAs per SM.  96 spiral / 36 cone-flat views: one volume, 3
// producers, 3 stages, 3 CTAs 3.54 / 3.07 ms; 2, 3, 3: 3.75 / 2.94; 4, 4, 2:
// 3.58 / 3.24; two volumes (twice the tile), 2, 3, 2: 4.72 / 4.09; 3, 3, 2:
// 4.68 / 4.51; 2, 2, 2: 5.87 / 4.91.
template <int NB> constexpr int kProd3 = NB == 1 ? 3 : 2;
template <int NB> constexpr int kFwdThreads3 = (kCons3 + kProd3<NB>) * 32;
template <int NB> constexpr int kStage3 = 3;
template <int NB> constexpr int kFwdMin3 = NB == 1 ? 3 : 2;
// (a producer must not wait for a stage two uses ahead of the consumers)
static_assert(kProd3<1> <= kStage3<1> && kProd3<2> <= kStage3<2>, "at least a stage per producer");
constexpr int kSeg = 16;     // column segments of one line held in shared memory
constexpr int kFast = 3;     // ... and held in registers by the usual path
constexpr int kZB = 16;      // slices of one copy
// pixels per slice of a tile: a CTA takes the narrowest that holds what its
// columns meet on any line (one tensor map each); most slices of a line in one
// step: the tile holds them and a neighbour at either end
constexpr int kNPitch = 7, kNarrow3 = 5;
__host__ __device__ constexpr int pitch3(int i) { return i < 3 ? 16 + 8 * i : i < 5 ? 16 * i : 32 * i - 64; }
__host__ __device__ constexpr int zwindow3(int pitch) { return pitch <= 64 ? 62 : 30; }
// bytes of a step's voxel tile: 64 slices of 64 pixels, 32 of 128
constexpr int kTileSlices3 = 64;
template <int NB> constexpr int kTileB3 = kTileSlices3 * 64 * 4 * NB;

// Tensor maps of the volumes' rows and columns (k_lines_of3): {pixel x
// volumes, line, slice, group}, boxes of one line, pitch3(i) pixels and kZB slices.
struct Maps3 {
    CUtensorMap m[2][kNPitch];   // [columns, rows][pitch]
};

struct Fwd3Args {
    dd_geom3d g;
    const char *plan;
    PlanLayout P;
    const float *volx, *volt;   // the volumes' rows and columns (k_lines_of3), from the launch's first volume
    float *out;          // (B, V, R, C)
    const float *sub;    // optional: out = A x - sub
    int *status;
    int V, nrb, ncg;     // views, row blocks, column groups
    int b0, geom, family;   // first volume of the launch; geometry and operator family
};

// A step of the forward kernel: one line, or some of its slices.
template <int NB>
struct Step3 {
    float4 h;                   // p0z, 1 / pintz, first slice, slices (0: nothing to do)
    int pitch, line;            // pixels per slice of the tile (0: no tile, the pixels are read from global memory)
    int fast, pad;              // tile present, no column with more than kFast segments, and the line in one step
    int nseg[kFC], j0[kFC];     // per column: segments (kSeg + 1: more), first pixel in the tile (on the line without one)
    float c[kSeg][kFC];         // coefficients
    float top[kTileSlices3];    // entry i: top of slice first + i - 1; +inf behind the last
};

// grid: (row block x group of 32 columns inside one walk block, view, volume
// group).  Lane = column, consumer warp w = rows r0 + RR w .. r0 + RR (w + 1) - 1.
//
// A line's part of a bin is separable: the overlaps of its column with the
// line's pixels (segments, the same for all rows) times the overlaps of its
// row with the slices.  So each consumer thread merges its RR rows with the
// slices in ascending z -- the slice that ends a row begins the next one --
// and sums the column's pixels once per slice it comes to, not once per row
// and slice; a step of the merge is an overlap of the two intervals and one
// multiply-add per volume.
//
// The producer warps turn line records (bulk copies, two in flight each) into
// segments and slice boundaries and start the tiled copies of the voxels the
// CTA's columns and rows can meet on the line (boxes of 16 slices) into one of
// kStage3 stages; full / empty mbarriers order them and the consumer warps,
// which run apart by up to a stage (no CTA barrier in the loop).
//
// Where the CTA's columns meet more pixels than its tile holds, the pixels are
// read from global memory by the step's segments; where a column meets more
// than kSeg, the consumers walk its record pixel by pixel.
//
// Bound by the latency of a merge's dependent steps at 20 to 33 warps an SM and by
// instruction issue (53 to 56 % of the slots, about 3,300 per line and CTA, a
// third of them the producers').  With every row's slices walked and
// each of its segments' voxels gathered from global memory it was about four
// times that.  2 x 256^3 cone beam, 36 views: 12.9 -> 4.1 ms; one 512 x 512 x
// 128 volume, 96 spiral views: 12.6 -> 3.5 ms.  On the way: the sums of all
// (column, slice) pairs formed first, lanes along z from global memory, 8.5 /
// 10.1 ms (7,100 instructions); per-slice bulk copies instead of boxes and the
// segments by the record walk, 5.0 / 7.2 ms.
// Columns of several pixels, ms by gathers per row and slice / by the record
// once per slice wherever the tile or 8 segments did not do / now: spiral,
// 512 x 512 x 128, 64 rows, 512 columns and 180 views 18.3 / 28.0 / 7.7, 256
// columns and 90 views 6.9 / 28.7 / 3.7; cone, 2 x 256^2 x 128, 128 rows, 60
// views, 128 columns 4.6 / 16.3 / 2.7; one 256^2 x 64, 64 rows, 60 views, 32
// columns 17.7 / 18.2 / 1.9, 16 columns 29.8 / 27.6 / 13.5.
template <int NB, int RR>
__global__ void __launch_bounds__(kFwdThreads3<NB>, kFwdMin3<NB>) k_fwd3(const __grid_constant__ Fwd3Args a, const __grid_constant__ Maps3 maps) {
    constexpr int kP = kProd3<NB>, kS = kStage3<NB>;
    using VT = Vox<NB>;
    using T = typename VT::T;
    extern __shared__ __align__(128) unsigned char sm[];   // [kS] voxel tiles
    const dd_geom3d &g = a.g;
    const int W = g.width, H = g.height, Dp = g.depth, C = g.num_col, R = g.num_row;
    const int v = blockIdx.y, cg = blockIdx.x % a.ncg, rb = blockIdx.x / a.ncg;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cc = (cg * kFC) / DD3_CHUNK, c0 = cc * DD3_CHUNK;
    const int k = cg * kFC + lane, kk = k - c0;
    const bool active = k < C;
    const bool prod = warp >= kCons3;   // the producer warps own no rows
    const int r0 = rb * (RR * kCons3) + warp * RR, b0 = a.b0 + blockIdx.z * NB;
    const PlanLayout &P = a.P;

    __shared__ __align__(128) DdLine srec[kP][2];
    __shared__ __align__(16) float4 slzr[kP][2];   // z quantities arriving with each record
    __shared__ __align__(16) Step3<NB> steps[kS];
    __shared__ float sdp[kFC + 1];
    __shared__ float zrange[kCons3 + 1][2];            // rows' z range per warp, and of the CTA
    __shared__ __align__(8) uint64_t full[kS], empty[kS], rbar[kP][2];
    __shared__ int abort_flag, armed[kS], nrec[kP][2];   // uses of the barriers so far

    __shared__ DdView3 w;
    if (tid < (int)(sizeof(DdView3) / sizeof(int)))
        reinterpret_cast<int *>(&w)[tid] = reinterpret_cast<const int *>(a.plan + P.views)[v * (int)(sizeof(DdView3) / sizeof(int)) + tid];
    const float *__restrict__ dpv = reinterpret_cast<const float *>(a.plan + P.dp) + (size_t)v * P.sdp;
    const float *__restrict__ rz = reinterpret_cast<const float *>(a.plan + P.rowz) + (size_t)v * P.srz;
    const float4 *__restrict__ linez = reinterpret_cast<const float4 *>(a.plan + P.linez) + (size_t)v * P.nl;
    const DdLine *__restrict__ lines = reinterpret_cast<const DdLine *>(a.plan + P.lines) + ((size_t)v * P.nch + cc) * P.nl;
    if (tid <= kFC) sdp[tid] = dpv[min(cg * kFC + tid, C)];
    if (tid == 0) {
        abort_flag = 0;
        for (int i = 0; i < kS; i++) {
            armed[i] = 0;
            dd_mbar_init(&full[i], 1);
            dd_mbar_init(&empty[i], kCons3);
        }
        for (int i = 0; i < kP; i++)
            for (int b = 0; b < 2; b++) {
                nrec[i][b] = 0;
                dd_mbar_init(&rbar[i][b], 1);
            }
        dd_fence_mbar_init();
    }
    __syncthreads();

    const int xb = w.xb;
    const int nline = xb ? H : W;

    // row boundaries; rows that do not exist (or are inverted) are empty
    // intervals where the previous row ended
    float rp0[RR], rp1[RR];
    {
        const float mag = active ? reinterpret_cast<const float *>(a.plan + P.mag)[(size_t)v * P.smag + k] : 1.0f;
        float zmin = 3.0e38f, zmax = -3.0e38f, last = 0.0f;
#pragma unroll
        for (int q = 0; q < RR; q++) {
            const int r = r0 + q;
            float e0 = 0.0f, e1 = 0.0f;
            if (active && !prod && r < R) dd3_rp(a.geom, &w, mag, rz[2 * r], rz[2 * r + 1], &e0, &e1);
            if (e0 < e1) {
                zmin = fminf(zmin, e0);
                zmax = fmaxf(zmax, e1);
                last = e1;
            } else {
                e0 = e1 = last;
            }
            rp0[q] = e0;
            rp1[q] = e1;
        }
        for (int o = 16; o > 0; o >>= 1) {
            zmin = fminf(zmin, __shfl_xor_sync(0xffffffffu, zmin, o));
            zmax = fmaxf(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
        }
        if (lane == 0 && !prod) {
            zrange[warp][0] = zmin;
            zrange[warp][1] = zmax;
        }
    }
    __syncthreads();
    if (tid == 0) {
        float lo = 3.0e38f, hi = -3.0e38f;
        for (int i = 0; i < kCons3; i++) {
            lo = fminf(lo, zrange[i][0]);
            hi = fmaxf(hi, zrange[i][1]);
        }
        zrange[kCons3][0] = lo;
        zrange[kCons3][1] = hi;
    }
    __syncthreads();

    // Steps per line: enough for the slices the CTA's rows can meet on the
    // line with the most of them; the tile's pitch: for the pixels its columns
    // meet on the line whose pixels are narrowest.  Both are an end of the
    // lines, unless the source lies between them (a negative pitch).
    constexpr int kAl = 4 / NB;   // pixels in 16 bytes
    int pi, zstep, nstep, nchunk;
    {
        const float zmin = zrange[kCons3][0], zmax = zrange[kCons3][1];
        const float4 la = linez[0], lb = linez[nline - 1];
        const float pm = fminf(la.z, lb.z), px = fminf(la.w / la.z, lb.w / lb.z), span = sdp[kFC] - sdp[0];
        const float widest = (pm > 0.0f && zmin < zmax) ? fminf((zmax - zmin) / pm + 4.0f, (float)Dp) : (float)Dp;
        const float npx = (pm > 0.0f && px > 0.0f && span >= 0.0f) ? span / px + (float)(2 + kAl) : 1.0e6f;
        // (tiles of more than 64 pixels only where they hold a line's slices at once)
        const int np = widest <= (float)zwindow3(pitch3(kNPitch - 1)) ? kNPitch : kNarrow3;
        for (pi = 0; pi < np - 1 && npx > (float)pitch3(pi); pi++) {}
        zstep = zwindow3(pitch3(pi));
        nchunk = max(1, ((int)widest + zstep - 1) / zstep);
        nstep = nline * nchunk;
    }
    const int tpitch = pitch3(pi);
    const int np4 = pad4(xb ? W : H);
    const T *__restrict__ src = reinterpret_cast<const T *>(xb ? a.volx : a.volt) + (size_t)blockIdx.z * Dp * nline * np4;

    if (prod) {
        const int p = warp - kCons3;
        auto issue = [&](int line, int buf) {   // a line's record (one lane)
            nrec[p][buf]++;
            dd_mbar_expect_tx(&rbar[p][buf], (uint32_t)(sizeof(DdLine) + sizeof(float4)));
            dd_bulk_g2s(&srec[p][buf], lines + line, (uint32_t)sizeof(DdLine), &rbar[p][buf]);
            dd_bulk_g2s(&slzr[p][buf], linez + line, (uint32_t)sizeof(float4), &rbar[p][buf]);
        };
        if (lane == 0) {
            if (p < nstep) issue(p / nchunk, 0);
            if (p + kP < nstep) issue((p + kP) / nchunk, 1);
        }
        const float zmin = zrange[kCons3][0], zmax = zrange[kCons3][1];
        const float dlo = sdp[lane], dhi = sdp[lane + 1];
        int st = p, use = 0, line = p / nchunk, part = p - line * nchunk;
        for (int m = p, n = 0; m < nstep; m += kP, n++) {
            const int buf = n & 1;
            bool ok = dd_mbar_wait(&rbar[p][buf], (uint32_t)(n >> 1) & 1u);
            if (ok && use > 0) ok = dd_mbar_wait(&empty[st], (uint32_t)(use - 1) & 1u);
            if (!__all_sync(0xffffffffu, ok)) {
                abort_flag = 1;
                break;
            }
            const DdLine *L = &srec[p][buf];
            const float4 lz = slzr[p][buf];
            Step3<NB> &S = steps[st];
            // slices [first, first + ns) of the step (a line behind the source
            // has a negative pitch and meets nothing)
            int first = 0, ns = 0;
            const float inv = 1.0f / lz.z;
            if (lz.z > 0.0f && zmin < zmax) {
                const float top = (float)Dp;
                first = (int)fminf(fmaxf(floorf((zmin - lz.x) * inv) - 1.0f, 0.0f), top);
                ns = (int)fminf(fmaxf(floorf((zmax - lz.x) * inv) + 2.0f, 0.0f), top) - first;
                const int skip = part * zstep;
                first += skip;
                ns = min(max(ns - skip, 0), zstep);
            }
            int nseg = 0, jb = 0, pitch = 0;
            bool fast = false;
            if (ns > 0) {
                for (int i = lane; i <= ns + 1; i += 32) {
                    float t = dd3_zb(lz.x, lz.z, first + i);
                    if (first + i == Dp) t = fminf(t, lz.y);
                    S.top[i] = (i == ns + 1) ? __int_as_float(0x7f800000) : t;
                }
                __syncwarp();
                // The column's segments: the lane's first pixel by a linear
                // estimate (the drift is a small part of a pixel), settled on
                // the exact boundaries; then the pixels in order.
                int jf = 0;
                const DdLineHdr hd = L->h;
                const float CL = (kk == hd.idet0) ? hd.bound0 : dlo, CH = dhi;
                if (active && hd.npiece > 0 && kk >= hd.idet0 && CL < CH) {
                    const DdPiece P0 = L->p[0];
                    const float t = floorf(FMUL(FSUB(CL, P0.Q), P0.invdl)) + (float)(P0.gb + 1);
                    int j = (int)fminf(fmaxf(t, (float)hd.i0), (float)(hd.nend - 1));
                    int pc = L->slot[dd_slot(CL)];
                    DdPiece Pc = L->p[pc];
                    auto bound = [&](int e) {   // boundary e >= i0; its piece is kept
                        while (pc < hd.npiece - 1 && e > Pc.gb) Pc = L->p[++pc];
                        while (pc > 0 && e <= L->p[pc - 1].gb) Pc = L->p[--pc];
                        return FADD(Pc.Q, FMUL((float)(e - Pc.gb), Pc.dl));
                    };
                    float plo = (j > hd.i0) ? bound(j - 1) : hd.bound0;
                    while (j > hd.i0 && plo > CL) {
                        j--;
                        plo = (j > hd.i0) ? bound(j - 1) : hd.bound0;
                    }
                    float phi = bound(j);
                    while (phi <= CL && j < hd.nend - 1) {
                        plo = phi;
                        phi = bound(++j);
                    }
                    jf = j;
                    plo = fmaxf(plo, CL);
                    if (phi > CL) {
                        const float lpos = (a.family == 2) ? dd3_line_pos_f(&g, &w, line) : 0.0f;
#pragma unroll 1
                        while (plo < CH) {
                            if (nseg == kSeg) {
                                nseg = kSeg + 1;
                                break;
                            }
                            S.c[nseg++][lane] = dd3_coef(a.geom, a.family, &g, &w, lpos, j, FSUB(fminf(phi, CH), plo), lz.w);
                            plo = phi;
                            if (++j >= hd.nend) break;
                            phi = bound(j);
                        }
                    }
                }
                const int lo = __reduce_min_sync(0xffffffffu, nseg > 0 ? jf : 0x7fffffff);
                const int hi = __reduce_max_sync(0xffffffffu, nseg > 0 ? jf + nseg : -1);
                const bool wide = __any_sync(0xffffffffu, nseg > kSeg);
                if (hi < 0) {
                    ns = 0;   // no column meets the line
                } else {
                    jb = lo / kAl * kAl;
                    pitch = tpitch;
                    if (wide || hi - jb > tpitch) jb = pitch = 0;
                }
                fast = __all_sync(0xffffffffu, nseg <= kFast) && pitch > 0 && nchunk == 1;
                S.nseg[lane] = nseg;
                S.j0[lane] = jf - jb;
            }
            if (lane == 0) {
                S.h = make_float4(lz.x, inv, __int_as_float(first), __int_as_float(ns));
                S.pitch = pitch;
                S.line = line;
                S.fast = fast;
            }
            __syncwarp();   // the record has been read, the step's arrays are written
            if (lane == 0) {
                // the voxels of slices first - 1 .. first + ns, in boxes of kZB
                // slices: the outer two are zero at the volume's ends, and
                // otherwise beyond the rows
                const int nbox = pitch > 0 ? (ns + 2 + kZB - 1) / kZB : 0;
                const uint32_t box_b = (uint32_t)(kZB * pitch * (int)sizeof(T));
                armed[st] = use + 1;
                dd_mbar_expect_tx(&full[st], box_b * (uint32_t)nbox);
                for (int i = 0; i < nbox; i++)
                    dd_tensor4_g2s(sm + st * kTileB3<NB> + i * box_b, &maps.m[xb][pi], jb * NB, line, first - 1 + i * kZB,
                                   (int)blockIdx.z, &full[st]);
                if (m + 2 * kP < nstep) issue(nchunk == 1 ? m + 2 * kP : (m + 2 * kP) / nchunk, buf);
            }
            st += kP;
            if (st >= kS) {
                st -= kS;
                use++;
            }
            for (part += kP; part >= nchunk; part -= nchunk) line++;
        }
    }

    T acc[RR];
#pragma unroll
    for (int q = 0; q < RR; q++) acc[q] = VT::zero();
    if (!prod) {
        int st = 0, par = 0;
        for (int m = 0; m < nstep; m++) {
            const bool ok = dd_mbar_wait(&full[st], (uint32_t)par);
            if (!__all_sync(0xffffffffu, ok)) {
                abort_flag = 1;
                break;
            }
            const Step3<NB> &S = steps[st];
            const float4 h = S.h;
            const int first = __float_as_int(h.z), n = __float_as_int(h.w), pitch = S.pitch;
            const int nseg = n > 0 ? S.nseg[lane] : 0;
            if (nseg > 0) {
                // entry (slice first + entry - 1) of the first row's lower
                // boundary: the closed-form estimate, settled on the exact boundaries
                int i = (int)fminf(fmaxf(floorf((rp0[0] - h.x) * h.y) - (float)(first - 1), 0.0f), (float)(n + 1));
                if (i > 0 && rp0[0] < S.top[i - 1]) i--;
                else if (i <= n && !(rp0[0] < S.top[i])) i++;
                const T *tile = reinterpret_cast<const T *>(sm + st * kTileB3<NB>) + S.j0[lane];   // entry 0
                const float *zp = S.top + i;
                if (S.fast) {   // uniform: the usual case, kept short
                    using K = typename VT::K;
                    const K k0 = VT::coef(S.c[0][lane]), k1 = VT::coef(S.c[1][lane]), k2 = VT::coef(S.c[2][lane]);   // unused past nseg
                    const bool p1 = nseg > 1, p2 = nseg > 2;
                    const T *r = tile + i * pitch;
                    auto column = [&]() -> T {
                        const T v0 = r[0], v1 = r[1], v2 = r[2];   // the tile is followed by room for these
                        T x = VT::kmul(k0, v0);
                        if (p1) x = VT::kfma(k1, v1, x);
                        if (p2) x = VT::kfma(k2, v2, x);
                        return x;
                    };
                    T x = column();
                    float zhi = *zp;
#pragma unroll
                    for (int q = 0; q < RR; q++) {
                        const float w0 = FSUB(fminf(rp1[q], zhi), rp0[q]);
                        if (w0 > 0.0f) acc[q] = VT::fma(w0, x, acc[q]);
                        while (zhi < rp1[q]) {   // so the next slice's overlap is positive
                            const float lo = zhi;
                            r += pitch;
                            x = column();
                            zhi = *++zp;
                            acc[q] = VT::fma(FSUB(fminf(rp1[q], zhi), lo), x, acc[q]);
                        }
                    }
                } else {
                    // rows and slices as above; column(e): the column's sum over entry e's pixels
                    auto merge = [&](auto column) {
                        int e = i;
                        T x = column(e);
                        float zhi = S.top[e];
#pragma unroll
                        for (int q = 0; q < RR; q++) {
                            const float w0 = FSUB(fminf(rp1[q], zhi), rp0[q]);
                            if (w0 > 0.0f) acc[q] = VT::fma(w0, x, acc[q]);
                            while (zhi < rp1[q]) {
                                const float lo = fmaxf(zhi, rp0[q]);
                                x = column(++e);
                                zhi = S.top[e];
                                const float w1 = FSUB(fminf(rp1[q], zhi), lo);
                                if (w1 > 0.0f) acc[q] = VT::fma(w1, x, acc[q]);
                            }
                        }
                    };
                    const int line = S.line;
                    const T *__restrict__ rows = src + ((size_t)(first - 1) * nline + line) * np4;   // entry 0's row
                    const size_t slice = (size_t)nline * np4;
                    if (nseg <= kSeg) {
                        const float *cs = &S.c[0][lane];
                        merge([&](int e) -> T {
                            T x = VT::zero();
                            if ((unsigned)(e - 1) >= (unsigned)n) return x;
                            if (pitch > 0) {
                                for (int t = 0; t < nseg; t++) x = VT::fma(cs[t * kFC], tile[e * pitch + t], x);
                                return x;
                            }
                            const T *__restrict__ r = rows + e * slice + S.j0[lane];
                            for (int t = 0; t < nseg; t += 4) {   // four loads in flight
                                T v[4];
#pragma unroll
                                for (int q = 0; q < 4; q++) v[q] = t + q < nseg ? __ldg(r + t + q) : VT::zero();
#pragma unroll
                                for (int q = 0; q < 4; q++)
                                    if (t + q < nseg) x = VT::fma(cs[(t + q) * kFC], v[q], x);
                            }
                            return x;
                        });
                    } else {   // more pixels than that: by the record, pixel by pixel
                        const DdLine *Lg = lines + line;
                        const float lpos = a.family == 2 ? dd3_line_pos_f(&g, &w, line) : 0.0f, parea = linez[line].w;
                        DdColWalk cw;
                        if (dd3_colwalk_init(Lg, sdp, lane, kk, &cw)) {
                            int j;
                            float wd;
                            while (dd3_colwalk_next(Lg, &cw, &j, &wd)) {
                                const float cf = dd3_coef(a.geom, a.family, &g, &w, lpos, j, wd, parea);
                                merge([&](int e) -> T {
                                    return (unsigned)(e - 1) < (unsigned)n ? VT::fma(cf, __ldg(rows + e * slice + j), VT::zero()) : VT::zero();
                                });
                            }
                        }
                    }
                }
            }
            __syncwarp();
            if (lane == 0) dd_mbar_arrive(&empty[st]);
            if (++st == kS) {
                st = 0;
                par ^= 1;
            }
        }
    }
    __syncthreads();
    if (abort_flag) {
        // let copies still in flight land before the CTA exits
        if (tid == 0) {
            for (int i = 0; i < kS; i++)
                if (armed[i] > 0) dd_mbar_drain(&full[i], (uint32_t)(armed[i] - 1) & 1u);
            for (int p = 0; p < kP; p++)
                for (int b = 0; b < 2; b++)
                    if (nrec[p][b] > 0) dd_mbar_drain(&rbar[p][b], (uint32_t)(nrec[p][b] - 1) & 1u);
            dd_report_timeout(a.status);
        }
        return;
    }
    if (!active || prod) return;
    const int ko = w.flip ? C - 1 - k : k;
#pragma unroll
    for (int q = 0; q < RR; q++) {
        const int r = r0 + q;
        if (r >= R) continue;
        float scale = w.bp_scale;
        if (a.family == 0) {
            float e0, e1;
            dd3_rp(a.geom, &w, reinterpret_cast<const float *>(a.plan + P.mag)[(size_t)v * P.smag + k], rz[2 * r],
                   rz[2 * r + 1], &e0, &e1);
            scale = dd3_proj_scale(&g, &w, sdp[lane], sdp[lane + 1], e0, e1);
        }
#pragma unroll
        for (int b = 0; b < NB; b++) {
            const size_t o = (((size_t)(b0 + b) * a.V + v) * R + r) * C + ko;
            float val = FMUL(VT::get(acc[q], b), scale);
            if (a.sub) val = FSUB(val, a.sub[o]);
            a.out[o] = val;
        }
    }
}

// ---------------------------------------------------------------------------
// Adjoint-type kernel: voxel gathers
// ---------------------------------------------------------------------------
struct Adj3Args {
    dd_geom3d g;
    const char *plan;
    PlanLayout P;
    const float *ss;     // pre-scaled sinogram, groups of (V, R, C, volumes), sorted columns
    float *out;          // (B, Dep, H, W)
    const float *base;   // optional: out = base + scale * value (may alias out)
    float scale;
    int *status;
    int B, V, ntx;
    int b0, family;      // first volume of the launch; operator family (dd3_coef)
};

// Shared memory of the adjoint kernel: buffers of one (view, walk block)'s data
// (the records of the tile's 16 lines, the block's column boundary and
// magnification tables, the row table, the lines' z quantities and the view
// record), each moved by bulk copies; all sizes are multiples of 16 bytes.
// kAdj3Bufs of them, or 2 where 3 row tables (8 bytes a row) do not fit.
constexpr int kAdj3Bufs = 3;
struct Adj3Smem {
    int rec, dp, mag, rz, lz, vw, bar, total;
    uint32_t rec_b, dp_b, mag_b, rz_b, lz_b;
};

__host__ __device__ inline Adj3Smem adj3_smem(const PlanLayout &P, int bufs) {
    Adj3Smem s;
    s.rec_b = (uint32_t)(kTile * sizeof(DdLine));
    s.dp_b = (uint32_t)((DD3_CHUNK + 4) * sizeof(float));
    s.mag_b = (uint32_t)(DD3_CHUNK * sizeof(float));
    s.rz_b = (uint32_t)(P.srz * sizeof(float));
    s.lz_b = (uint32_t)(kTile * sizeof(float4));
    int o = 0;
    s.rec = o; o += bufs * (int)s.rec_b;
    s.dp = o; o += bufs * (int)s.dp_b;
    s.mag = o; o += bufs * (int)s.mag_b;
    s.rz = o; o += bufs * (int)s.rz_b;
    s.lz = o; o += bufs * (int)s.lz_b;
    s.vw = o; o += bufs * (int)sizeof(DdView3);
    s.bar = o; o += bufs * (int)sizeof(uint64_t);
    s.total = (o + 127) & ~127;
    return s;
}

// The size limit of a view's tables: what two buffers of a whole view (all its
// walk blocks) take beside 200 KB.  Two of the adjoint's buffers, which hold one
// block each, fit whatever passes it.
inline bool view_too_wide(const PlanLayout &P, int R) {
    const size_t one = (size_t)kTile * P.nch * sizeof(DdLine) + sizeof(float) * ((size_t)P.sdp + P.smag + pad4(2 * R)) +
                       kTile * sizeof(float4) + sizeof(DdView3) + sizeof(uint64_t);
    return (2 * one + 127) / 128 * 128 > 200 * 1024;
}

// Can view w see the slab of slices [s0, s0 + ns) on the walked lines
// l0..l1 (with one slice of margin)?
__device__ __forceinline__ bool slab_visible(const dd_geom3d &g, const DdView3 &w, int l0, int l1, int s0,
                                             int ns, float zr0, float zr1) {
    const float m0 = dd3_line_mag(&w, dd3_line_pos_f(&g, &w, l0));
    const float m1 = dd3_line_mag(&w, dd3_line_pos_f(&g, &w, l1));
    const float zsA = w.z0 + (float)(s0 - 1) * g.pix_z, zsB = w.z0 + (float)(s0 + ns + 1) * g.pix_z;
    return dd3_slab_lit(&w, fminf(m0, m1), fmaxf(m0, m1), zsA, zsB, zr0, zr1);
}

// Plan time: for each slab of kZS slices, the views [first, last] whose
// detector can see it anywhere in the image -- slab_visible over the whole
// image's lines, a superset of what it admits for any tile's lines (wider
// magnification bounds only widen the lit band) -- stored as {first,
// last + 1}, {0, 0} if none.  The adjoint loops over these views only: on a
// spiral a slab is lit during one pass of the helix.
__global__ void __launch_bounds__(256) k_slab_views3(dd_geom3d g, char *plan, PlanLayout P, int V) {
    const int slab = blockIdx.x, R = g.num_row;
    const DdView3 *views = reinterpret_cast<const DdView3 *>(plan + P.views);
    const float *rzt = reinterpret_cast<const float *>(plan + P.rowz);
    __shared__ int lo, hi;
    if (threadIdx.x == 0) {
        lo = V;
        hi = -1;
    }
    __syncthreads();
    int mylo = V, myhi = -1;
    for (int v = threadIdx.x; v < V; v += blockDim.x) {
        const DdView3 w = views[v];
        const int nline = w.xb ? g.height : g.width;
        const float *rzv = rzt + (size_t)v * P.srz;
        if (slab_visible(g, w, 0, nline - 1, slab * kZS, kZS, rzv[0], rzv[2 * R - 1])) {
            mylo = min(mylo, v);
            myhi = max(myhi, v);
        }
    }
    atomicMin(&lo, mylo);
    atomicMax(&hi, myhi);
    __syncthreads();
    if (threadIdx.x == 0)
        reinterpret_cast<int2 *>(plan + P.slabv)[slab] = hi >= lo ? make_int2(lo, hi + 1) : make_int2(0, 0);
}

// grid: (voxel-column tile, ZS slices, volume group); thread = one (x, y)
// voxel column of a 16 x 16 tile.
//
// The work is a list of units (view, walk block of 256 columns).  Every 32
// views each lane of a warp looks at one of them: whether its detector sees
// the slab, which walk blocks the tile's shadow touches (one, or two where it
// straddles a boundary), and the column grid linearised around the tile --
// so views that miss the tile cost nothing, and a unit's records and tables
// are all that is staged (three buffers, one CTA barrier per unit).
//
// Per segment (pixel, detector column) the thread walks its slices and the
// column's rows together, in ascending z: the row that ends a slice is the
// first candidate of the next one, so every row is projected (dd3_rp) and
// loaded once per segment, and a step is an overlap of the two intervals and
// one multiply-add per volume.
//
// Bound by the loads of the sinogram inside that walk (long scoreboard is the first
// stall; 54 to 60 % of the issue slots are used) and by finding each pixel's columns
// and boundaries, which ZS slices share.  One 512 x 512 x 128 volume, 1140
// spiral views: 317 ms with a row search per slice, every walk block of every
// view staged and searched, and 8 slices a thread; 192 ms with the carried
// row walk alone; 108 ms with the unit list, the linear column estimate and
// 16 slices.  2 x 256^3 cone beam, 360 views: 145, 63, 49 ms.
template <int GEOM, int NB, int ZS, int BUFS>
__global__ void __launch_bounds__(kThreads, 3) k_adj3(const Adj3Args a) {
    using VT = Vox<NB>;
    using T = typename VT::T;
    extern __shared__ __align__(128) unsigned char sm[];
    const dd_geom3d &g = a.g;
    const int W = g.width, H = g.height, Dp = g.depth, C = g.num_col, R = g.num_row;
    const PlanLayout &P = a.P;
    const Adj3Smem S = adj3_smem(P, BUFS);
    const int tid = threadIdx.x, lane = tid & 31;
    const int tX = blockIdx.x % a.ntx, tY = blockIdx.x / a.ntx;
    const int xlo = tX * kTile, ylo = tY * kTile;
    const int x = xlo + (tid & (kTile - 1)), y = ylo + (tid / kTile);
    const bool active = x < W && y < H;
    const int s0 = blockIdx.y * ZS, b0 = a.b0 + blockIdx.z * NB;
    const DdView3 *__restrict__ views = reinterpret_cast<const DdView3 *>(a.plan + P.views);
    const float *__restrict__ dpt = reinterpret_cast<const float *>(a.plan + P.dp);
    const float *__restrict__ magt = reinterpret_cast<const float *>(a.plan + P.mag);
    const float *__restrict__ rzt = reinterpret_cast<const float *>(a.plan + P.rowz);
    const float4 *__restrict__ linez = reinterpret_cast<const float4 *>(a.plan + P.linez);
    const DdLine *__restrict__ lines = reinterpret_cast<const DdLine *>(a.plan + P.lines);
    const size_t per = (size_t)a.V * R * C;
    const T *__restrict__ ssb = reinterpret_cast<const T *>(a.ss + (size_t)b0 * per);
    const int family = a.family;
    uint64_t *bar = reinterpret_cast<uint64_t *>(sm + S.bar);
    __shared__ int abort_flag;

    if (tid == 0) {
        abort_flag = 0;
        for (int i = 0; i < BUFS; i++) dd_mbar_init(&bar[i], 1);
        dd_fence_mbar_init();
    }
    __syncthreads();

    // a unit's copies (one thread)
    auto issue = [&](int v, int cc, int buf) {
        const int xbv = views[v].xb;
        const int l0 = xbv ? ylo : xlo;
        const int n = min(kTile, (xbv ? H : W) - l0);
        const int c0 = cc * DD3_CHUNK;
        const uint32_t rb = (uint32_t)(n * sizeof(DdLine)), lb = (uint32_t)(n * sizeof(float4));
        const uint32_t db = (uint32_t)(min(DD3_CHUNK + 4, P.sdp - c0) * sizeof(float));
        const uint32_t mb = (uint32_t)(min(DD3_CHUNK, P.smag - c0) * sizeof(float));
        dd_mbar_expect_tx(&bar[buf], rb + db + mb + S.rz_b + lb + (uint32_t)sizeof(DdView3));
        dd_bulk_g2s(sm + S.rec + buf * S.rec_b, lines + ((size_t)v * P.nch + cc) * P.nl + l0, rb, &bar[buf]);
        dd_bulk_g2s(sm + S.dp + buf * S.dp_b, dpt + (size_t)v * P.sdp + c0, db, &bar[buf]);
        dd_bulk_g2s(sm + S.mag + buf * S.mag_b, magt + (size_t)v * P.smag + c0, mb, &bar[buf]);
        dd_bulk_g2s(sm + S.rz + buf * S.rz_b, rzt + (size_t)v * P.srz, S.rz_b, &bar[buf]);
        dd_bulk_g2s(sm + S.lz + buf * S.lz_b, linez + (size_t)v * P.nl + l0, lb, &bar[buf]);
        dd_bulk_g2s(sm + S.vw + buf * (int)sizeof(DdView3), views + v, (uint32_t)sizeof(DdView3), &bar[buf]);
    };

    // the views that can see the CTA's slices somewhere in the image
    int2 vr = make_int2(a.V, 0);
    for (int q = 0; q < ZS / kZS; q++) {
        const int slab = s0 / kZS + q;
        if (slab >= P.nslab) break;
        const int2 r = reinterpret_cast<const int2 *>(a.plan + P.slabv)[slab];
        if (r.x < r.y) {
            vr.x = min(vr.x, r.x);
            vr.y = max(vr.y, r.y);
        }
    }
    const int ns = min(ZS, Dp - s0);

    // The list of units, kept by the first warp: `next` writes one more (v < 0
    // past the last) into its slot.  The lanes' views and what is known of
    // them wait in shared memory, so that the walk below has the registers.
    struct Unit {
        int v, cc;
        float A, B;   // column of axis position u: about A u + B
    };
    __shared__ Unit units[4];
    __shared__ float la_s[32], lb_s[32];
    __shared__ int cc_s[32];   // walk blocks of the lane's view: first | last << 16
    int vbase = vr.x - 32, ccn = 0, cce = -1;   // next and last block of the current view
    unsigned mask = 0;
    int cur = 0;
    auto next = [&](Unit *u) {
        while (ccn > cce) {
            while (mask == 0) {
                vbase += 32;
                if (vbase >= vr.y) {
                    if (lane == 0) u->v = -1;
                    vbase = vr.y;
                    __syncwarp();
                    return;
                }
                const int v = vbase + lane;
                bool lit = false;
                if (v < vr.y) {
                    const DdView3 w = views[v];
                    const float *rzv = rzt + (size_t)v * P.srz;
                    const int l0 = w.xb ? ylo : xlo, l1 = min(l0 + kTile, w.xb ? H : W) - 1;
                    lit = slab_visible(g, w, l0, l1, s0, ns, rzv[0], rzv[2 * R - 1]);
                    if (lit) {
                        // the tile's shadow on the axis: its four corners
                        const float *dpv = dpt + (size_t)v * P.sdp;
                        const float X0 = ((float)xlo - 0.5f * (float)W) * g.pix_x + g.pix_xshift;
                        const float X1 = ((float)min(xlo + kTile, W) - 0.5f * (float)W) * g.pix_x + g.pix_xshift;
                        const float Y0 = (0.5f * (float)H - (float)ylo) * g.pix_y + g.pix_yshift;
                        const float Y1 = (0.5f * (float)H - (float)min(ylo + kTile, H)) * g.pix_y + g.pix_yshift;
                        const float src = w.xb ? w.srcy : w.srcx;
                        const float d0 = (w.xb ? Y0 : X0) - src, d1 = (w.xb ? Y1 : X1) - src;
                        float lo = 3.0e38f, hi = -3.0e38f;
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const float px = (i & 1) ? X1 : X0, py = (i & 2) ? Y1 : Y0;
                            const float t = w.xb ? dd_map2x(w.srcx, w.srcy, px, py) : dd_map2y(w.srcx, w.srcy, px, py);
                            lo = fminf(lo, t);
                            hi = fmaxf(hi, t);
                        }
                        int ca = 0, cb = P.nch - 1;
                        float la = 0.0f, lb = 0.0f;
                        if (d0 * d1 > 0.0f && lo <= hi) {   // the source's line does not cross the tile
                            const float tol = 0.0625f * (hi - lo) + 1e-4f * (fabsf(lo) + fabsf(hi));   // a pixel, and the drift
                            while (ca < cb) {   // blocks that end below the shadow
                                const float e = dpv[(ca + 1) * DD3_CHUNK];
                                if (!(e >= dpv[ca * DD3_CHUNK] && e < lo - tol)) break;
                                ca++;
                            }
                            while (cb > ca) {   // blocks that start above it
                                const float b = dpv[cb * DD3_CHUNK];
                                if (!(b > hi + tol && b <= dpv[min((cb + 1) * DD3_CHUNK, C)])) break;
                                cb--;
                            }
                            const float um = 0.5f * (lo + hi);
                            const int k = min(dd3_col_of(GEOM, &g, &w, dpv, um, 0, C), C - 1);
                            const float b = dpv[k], e = dpv[k + 1];
                            if (e > b) {
                                la = __fdividef(1.0f, e - b);
                                lb = (float)k - b * la;
                            }
                        }
                        la_s[lane] = la;
                        lb_s[lane] = lb;
                        cc_s[lane] = ca | (cb << 16);
                    }
                }
                mask = __ballot_sync(0xffffffffu, lit);
            }
            __syncwarp();
            cur = __ffs(mask) - 1;
            mask &= mask - 1;
            ccn = cc_s[cur] & 0xFFFF;
            cce = cc_s[cur] >> 16;
        }
        if (lane == 0) *u = Unit{vbase + cur, ccn, la_s[cur], lb_s[cur]};
        ccn++;
        __syncwarp();
    };

    T acc[ZS];
#pragma unroll
    for (int q = 0; q < ZS; q++) acc[q] = VT::zero();

    DdPhases ph;
    // unit i uses buffer i % BUFS; the BUFS - 1 units behind it are in flight
    constexpr int ahead = BUFS - 1;
    if (tid < 32) {
        next(&units[0]);
        if (ahead > 1) next(&units[1]);
        if (tid == 0) {
            if (units[0].v >= 0) issue(units[0].v, units[0].cc, 0);
            if (ahead > 1 && units[1].v >= 0) issue(units[1].v, units[1].cc, 1);
        }
    }
    __syncthreads();
    int buf = 0;
    for (int i = 0; units[i & 3].v >= 0; i++, buf = buf == ahead ? 0 : buf + 1) {
        const int buf2 = buf == 0 ? ahead : buf - 1;   // buffer of unit i + ahead (and of unit i - 1)
        // slot i + ahead was last read before the barrier of unit i - 1
        if (tid < 32) next(&units[(i + ahead) & 3]);
        if (!dd_mbar_wait(&bar[buf], ph.parity(buf))) abort_flag = 1;
        ph.flip(buf);
        // past this barrier every warp has finished unit i - 1
        __syncthreads();
        if (abort_flag) {
            // this unit's copies (the wait gave up on them) and, of three buffers, the next one's may be in flight
            if (tid == 0) {
                const int b1 = buf == ahead ? 0 : buf + 1;
                dd_mbar_drain(&bar[buf], ph.parity(buf) ^ 1u);
                if (ahead > 1 && units[(i + 1) & 3].v >= 0) dd_mbar_drain(&bar[b1], ph.parity(b1));
            }
            break;
        }
        if (tid == 0 && units[(i + ahead) & 3].v >= 0) issue(units[(i + ahead) & 3].v, units[(i + ahead) & 3].cc, buf2);
        const DdView3 &w = *reinterpret_cast<const DdView3 *>(sm + S.vw + buf * (int)sizeof(DdView3));
        const int xb = w.xb;
        const int rl = xb ? (y - ylo) : (x - xlo);
        const int j = xb ? x : H - 1 - y;
        const DdLine *L = reinterpret_cast<const DdLine *>(sm + S.rec + buf * S.rec_b) + rl;
        const float4 lz = reinterpret_cast<const float4 *>(sm + S.lz + buf * S.lz_b)[rl];
        const Unit u0 = units[i & 3];
        const int c0 = u0.cc * DD3_CHUNK;
        float PL, PH;
        // (a line behind the source has a negative pitch and meets nothing)
        if (active && lz.z > 0.0f && dd3_pix_bounds(L, j, &PL, &PH)) {
            const float *dp = reinterpret_cast<const float *>(sm + S.dp + buf * S.dp_b);     // from column c0
            const float *mg = reinterpret_cast<const float *>(sm + S.mag + buf * S.mag_b);
            const float2 *rz = reinterpret_cast<const float2 *>(sm + S.rz + buf * S.rz_b);
            const int klo = L->h.idet0, khi = min(DD3_CHUNK, C - c0);
            const float lpos = (family == 2) ? dd3_line_pos_f(&g, &w, (xb ? ylo : xlo) + rl) : 0.0f;
            const float srcz = (GEOM == DD_GEOM3_SPIRAL) ? w.srcz : 0.0f;
            auto row_z = [&](float mag, float2 z, float *e0, float *e1) {   // dd3_rp
                if (GEOM == DD_GEOM3_SPIRAL) {
                    *e0 = FADD(FMUL(mag, FSUB(z.x, srcz)), srcz);
                    *e1 = FADD(FMUL(mag, FSUB(z.y, srcz)), srcz);
                } else {
                    *e0 = FMUL(mag, z.x);
                    *e1 = FMUL(mag, z.y);
                }
            };
            // past the volume's top the slice boundaries coincide, so those
            // slices meet no row
            const float ztop = fminf(dd3_zb(lz.x, lz.z, Dp), lz.y);
            const float zfirst = dd3_zb(lz.x, lz.z, s0);
            const T *__restrict__ ssv = ssb + (size_t)u0.v * R * C + c0;
            int k = klo;
            float CL = L->h.bound0;
            if (dp[khi] > PL) {
                // first column that ends above the pixel's lower boundary:
                // the linear estimate, settled on the exact boundaries
                k = max(klo, min(khi - 1, (int)floorf(fminf(fmaxf(fmaf(PL, u0.A, u0.B), 0.0f), 1.0e6f)) - c0));
                while (k > klo && dp[k] > PL) k--;
                while (k < khi && dp[k + 1] <= PL) k++;
                if (k > klo) CL = dp[k];
            } else {
                k = khi;
            }
            for (; k < khi && CL < PH; k++) {
                const float CH = dp[k + 1];
                const float wd = FSUB(fminf(PH, CH), fmaxf(PL, CL));
                CL = CH;
                const float mag = mg[k];
                if (!(wd > 0.0f && mag > 0.0f)) continue;
                const float coef = dd3_coef(GEOM, family, &g, &w, lpos, j, wd, lz.w);
                // first row that reaches above the first slice's bottom: the
                // closed-form estimate, settled on the exact boundaries
                // (row R lies at infinity and ends the walk)
                const float zeta = dd3_approx_div(zfirst - srcz, mag) + srcz;
                int r = (int)floorf(fminf(fmaxf((zeta - w.rzA) * w.rzI, 0.0f), (float)(R - 1)));
                float e0, e1;
                row_z(mag, rz[r], &e0, &e1);
                while (!(e1 > zfirst) && r < R) row_z(mag, rz[++r], &e0, &e1);
                while (r > 0 && e0 > zfirst) row_z(mag, rz[--r], &e0, &e1);
                if (r >= R) continue;
                const T *__restrict__ p = ssv + (size_t)r * C + k;
                T val = __ldg(p);
                float hi = zfirst;
#pragma unroll
                for (int q = 0; q < ZS; q++) {
                    const float lo = hi;
                    hi = fminf(dd3_zb(lz.x, lz.z, s0 + q + 1), ztop);
                    T t = VT::zero();
                    const float w0 = FSUB(fminf(e1, hi), fmaxf(e0, lo));
                    if (w0 > 0.0f) t = VT::fma(w0, val, t);
                    while (e1 < hi) {
                        row_z(mag, rz[++r], &e0, &e1);
                        p += C;
                        if (r < R) val = __ldg(p);
                        const float w1 = FSUB(fminf(e1, hi), e0);
                        if (w1 > 0.0f) t = VT::fma(w1, val, t);
                    }
                    acc[q] = VT::fma(coef, t, acc[q]);
                }
            }
        }
    }
    if (abort_flag) {
        if (tid == 0) dd_report_timeout(a.status);
        return;
    }
    if (!active) return;
#pragma unroll
    for (int q = 0; q < ZS; q++) {
        const int s = s0 + q;
        if (s >= Dp) continue;
#pragma unroll
        for (int b = 0; b < NB; b++) {
            const size_t o = (((size_t)(b0 + b) * Dp + s) * H + y) * W + x;
            const float val = VT::get(acc[q], b);
            a.out[o] = a.base ? fmaf(a.scale, val, a.base[o]) : val;
        }
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
int geom_of(int scan) {
    return scan == DD_SCAN_CONE_FLAT ? DD_GEOM3_CONE_FLAT : (scan == DD_SCAN_CONE_ARC ? DD_GEOM3_CONE_ARC : DD_GEOM3_SPIRAL);
}

int validate(int scan, int op, const dd_geom3d *g, int B, int V) {
    if (!g) return DD_ERR_INVALID_ARG;
    if (scan < DD_SCAN_CONE_FLAT || scan > DD_SCAN_SPIRAL) return DD_ERR_INVALID_ARG;
    if (op < DD_OP_PROJ || op > DD_OP_BPROJ_TW) return DD_ERR_INVALID_ARG;
    if (g->width <= 0 || g->height <= 0 || g->depth <= 0 || g->num_col <= 0 || g->num_row <= 0 || B <= 0 ||
        V <= 0)
        return DD_ERR_INVALID_ARG;
    const float f[] = {g->pix_x, g->pix_y, g->pix_z, g->col_size, g->row_size, g->iso_source,
                       g->source_detector, g->pix_xshift, g->pix_yshift, g->pix_zshift, g->col_shift,
                       g->row_shift};
    for (float x : f)
        if (!(x == x) || x - x != 0.0f) return DD_ERR_INVALID_ARG;   // NaN / inf
    if (!(g->pix_x > 0 && g->pix_y > 0 && g->pix_z > 0 && g->col_size > 0 && g->row_size > 0))
        return DD_ERR_INVALID_ARG;
    if (!(g->iso_source > 0 && g->source_detector > 0)) return DD_ERR_INVALID_ARG;
    const long long lim = (1LL << 31) - 1;
    if ((long long)g->width * g->height * g->depth * B > lim) return DD_ERR_SIZE_OVERFLOW;
    if ((long long)V * g->num_row * g->num_col * B > lim) return DD_ERR_SIZE_OVERFLOW;
    if (g->width > 8192 || g->height > 8192 || V > 65535 || g->num_row > 65535 || g->num_col > 65535)
        return DD_ERR_SIZE_OVERFLOW;
    if (view_too_wide(plan_layout(g, V), g->num_row)) return DD_ERR_SIZE_OVERFLOW;
    return DD_OK;
}

int launch_status() {
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? DD_OK : DD_ERR_LAUNCH;
}

int plan(int scan, const dd_geom3d *g, const float *angles, const float *sp, int V, void *planp, size_t bytes,
         cudaStream_t st) {
    const PlanLayout P = plan_layout(g, V);
    if (!planp || bytes < P.total) return DD_ERR_WORKSPACE;
    if (!angles || (scan == DD_SCAN_SPIRAL && !sp)) return DD_ERR_INVALID_ARG;
    char *base = (char *)planp;
    const int geom = geom_of(scan);
    dd2::ProfRec *pr = dd2::prof_begin(DD_KERNEL_PLAN, st);
    const dim3 gl((unsigned)((P.nl * P.nch + 127) / 128), (unsigned)V);
    if (geom == DD_GEOM3_CONE_FLAT) {
        k_views3<DD_GEOM3_CONE_FLAT><<<V, kThreads, 0, st>>>(*g, angles, sp, V, base, P);
        k_lines3<DD_GEOM3_CONE_FLAT><<<gl, 128, 0, st>>>(*g, base, P);
    } else if (geom == DD_GEOM3_CONE_ARC) {
        k_views3<DD_GEOM3_CONE_ARC><<<V, kThreads, 0, st>>>(*g, angles, sp, V, base, P);
        k_lines3<DD_GEOM3_CONE_ARC><<<gl, 128, 0, st>>>(*g, base, P);
    } else {
        k_views3<DD_GEOM3_SPIRAL><<<V, kThreads, 0, st>>>(*g, angles, sp, V, base, P);
        k_lines3<DD_GEOM3_SPIRAL><<<gl, 128, 0, st>>>(*g, base, P);
    }
    k_slab_views3<<<P.nslab, 256, 0, st>>>(*g, base, P, V);
    dd2::prof_end(pr, st);
    dd2::count_launches(3);
    return launch_status();
}

// cuTensorMapEncodeTiled, from the driver the runtime has loaded
using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled() {
    static const EncodeTiled fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            (void)cudaGetLastError();
            p = nullptr;
        }
        return (EncodeTiled)p;
    }();
    return fn;
}

template <int NB>
int make_maps3(const Fwd3Args &a, int ngroups, Maps3 *maps) {
    const EncodeTiled enc = encode_tiled();
    if (!enc) return DD_ERR_LAUNCH;
    for (int rows = 0; rows < 2; rows++) {
        const cuuint64_t np = (cuuint64_t)(rows ? a.g.width : a.g.height), nl = (cuuint64_t)(rows ? a.g.height : a.g.width);
        const cuuint64_t line_b = (cuuint64_t)pad4((int)np) * NB * sizeof(float);
        const cuuint64_t dim[4] = {np * NB, nl, (cuuint64_t)a.g.depth, (cuuint64_t)ngroups};
        const cuuint64_t str[3] = {line_b, line_b * nl, line_b * nl * dim[2]};
        const cuuint32_t one[4] = {1, 1, 1, 1};
        for (int i = 0; i < kNPitch; i++) {
            const cuuint32_t box[4] = {(cuuint32_t)(pitch3(i) * NB), 1, kZB, 1};
            if (enc(&maps->m[rows][i], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (void *)(rows ? a.volx : a.volt), dim, str, box,
                    one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return DD_ERR_LAUNCH;
        }
    }
    return DD_OK;
}

template <int NB, int RR>
int launch_fwd_rows(Fwd3Args a, int ngroups, cudaStream_t st) {
    a.ncg = (a.g.num_col + kFC - 1) / kFC;
    a.nrb = (a.g.num_row + RR * kCons3 - 1) / (RR * kCons3);
    const long long nx = (long long)a.ncg * a.nrb;
    if (nx > 0x7FFFFFFFLL) return DD_ERR_SIZE_OVERFLOW;
    const int smem = kStage3<NB> * kTileB3<NB> + kFast * 8;   // the fast path reads up to two pixels past a row
    if (cudaFuncSetAttribute(k_fwd3<NB, RR>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
        return DD_ERR_LAUNCH;
    Maps3 maps;
    const int rc = make_maps3<NB>(a, ngroups, &maps);
    if (rc != DD_OK) return rc;
    k_fwd3<NB, RR><<<dim3((unsigned)nx, (unsigned)a.V, (unsigned)ngroups), kFwdThreads3<NB>, smem, st>>>(a, maps);
    dd2::count_launches(1);
    return DD_OK;
}

// Rows per thread: 8, 4 or 2, whichever leaves least work for rows that do not
// exist -- a step costs a thread its rows plus about 2.5 rows' worth of
// finding the first slice and of its share of the producers -- or for SMs that
// get no CTA: where CTAs do not fill the chip (3 per SM with one volume, 2 with
// two) fewer rows are more CTAs.  128 x 128 x 64, 24 views, 200 x 64 cells, 1 /
// 2 / 3 volumes: 0.60 / 0.54 / 1.15 ms with 8 rows, 0.18 / 0.26 / 0.44 with 4.
// Rows that meet more slices than a step holds take each line in parts, without
// the usual path's registers: at least twice the time.  224 x 224 x 200, 60
// views, 300 x 180 cells, 1 / 2 volumes: 6.7 / 7.2 ms with 8 rows, 2.1 / 2.8
// with 4.  Where 32 columns meet more than 64 pixels on some views, rows that
// meet more slices than a tile of 128 pixels holds gather from global memory
// there: 1.3 times (spiral, 512 x 512 x 128, 64 rows, 512 columns and 180 views /
// 256 columns and 90 views: 11.5 / 9.7 ms with 8 rows, 7.7 / 3.7 with 4).
template <int NB>
int launch_fwd_volumes(Fwd3Args a, int b0, int ngroups, cudaStream_t st) {
    if (ngroups <= 0) return DD_OK;
    a.b0 = b0;
    a.volx += (size_t)b0 * a.g.depth * a.g.height * pad4(a.g.width);
    a.volt += (size_t)b0 * a.g.depth * a.g.width * pad4(a.g.height);
    const int R = a.g.num_row;
    const double full = 152.0 * kFwdMin3<NB>, per_block = (double)((a.g.num_col + kFC - 1) / kFC) * a.V * ngroups;
    // slices the rows of a CTA meet on the farthest line
    const double row_slices = a.g.row_size * (a.g.iso_source + 0.6 * std::max(a.g.width * a.g.pix_x, a.g.height * a.g.pix_y)) /
                              (a.g.source_detector * a.g.pix_z);
    // pixels its columns meet there, on views halfway to 45 degrees
    const double cell = a.geom == DD_GEOM3_CONE_FLAT ? a.g.col_size * a.g.iso_source / a.g.source_detector : a.g.col_size * a.g.iso_source;
    const double far = 1.0 + 0.6 * std::max(a.g.width * a.g.pix_x, a.g.height * a.g.pix_y) / a.g.iso_source;
    const bool wide = 1.15 * kFC * cell * far / std::min(a.g.pix_x, a.g.pix_y) + 3 > pitch3(kNarrow3 - 1);
    const int most = zwindow3(pitch3(kNarrow3 - 1)), few = zwindow3(pitch3(kNPitch - 1));
    auto cost = [&](int rr) {
        const double blocks = std::max(((R + rr * kCons3 - 1) / (rr * kCons3)) * per_block, full);
        const double meet = std::min(R, rr * kCons3) * row_slices + 4;
        const bool parts = a.g.depth > most && meet > most, gather = wide && a.g.depth > few && meet > few;
        return blocks * (rr + 2.5) * (parts ? 2 : 1) * (gather ? 1.3 : 1);
    };
    const double c8 = cost(8), c4 = cost(4), c2 = cost(2);
    if (c8 <= c4 && c8 <= c2) return launch_fwd_rows<NB, 8>(a, ngroups, st);
    if (c4 <= c2) return launch_fwd_rows<NB, 4>(a, ngroups, st);
    return launch_fwd_rows<NB, 2>(a, ngroups, st);
}

template <int GEOM, int NB, int ZS, int BUFS>
int launch_adj_slabs(const Adj3Args &a, int ngroups, cudaStream_t st) {
    const int smem = adj3_smem(a.P, BUFS).total;
    auto kern = k_adj3<GEOM, NB, ZS, BUFS>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return DD_ERR_LAUNCH;
    const int nty = (a.g.height + kTile - 1) / kTile;
    const dim3 grid((unsigned)(a.ntx * nty), (unsigned)((a.g.depth + ZS - 1) / ZS), (unsigned)ngroups);
    kern<<<grid, kThreads, smem, st>>>(a);
    dd2::count_launches(1);
    return DD_OK;
}

// 16 slices per thread share a pixel's columns and boundaries; 8 where 16
// would leave the chip's 456 resident CTAs (3 per SM) less than twice full.
// Detectors whose row tables leave no room for three buffers (1 KB is for the
// kernel's static arrays) take two, 8 slices a thread.
template <int GEOM, int NB>
int launch_adj_kernel(Adj3Args a, int b0, int ngroups, cudaStream_t st) {
    if (ngroups <= 0) return DD_OK;
    a.b0 = b0;
    if (adj3_smem(a.P, kAdj3Bufs).total + 1024 > 227 * 1024) return launch_adj_slabs<GEOM, NB, kZS, 2>(a, ngroups, st);
    const long long tiles = (long long)a.ntx * ((a.g.height + kTile - 1) / kTile) * ngroups;
    if (tiles * ((a.g.depth + 2 * kZS - 1) / (2 * kZS)) >= 2 * 456)
        return launch_adj_slabs<GEOM, NB, 2 * kZS, kAdj3Bufs>(a, ngroups, st);
    return launch_adj_slabs<GEOM, NB, kZS, kAdj3Bufs>(a, ngroups, st);
}

template <int GEOM>
int launch_adj(const Adj3Args &a, const float *in, float *ss, cudaStream_t st) {
    const dd_geom3d &g = a.g;
    const dim3 gs((unsigned)((g.num_col + 127) / 128), (unsigned)g.num_row, (unsigned)a.V);
    dd2::ProfRec *pt = dd2::prof_begin(DD_KERNEL_TABLES, st);
    if (a.family == 0) k_sino3<GEOM, 0><<<gs, 128, 0, st>>>(g, a.plan, a.P, in, ss, a.B, a.V, a.status);
    else k_sino3<GEOM, 1><<<gs, 128, 0, st>>>(g, a.plan, a.P, in, ss, a.B, a.V, a.status);
    dd2::prof_end(pt, st);
    dd2::count_launches(1);
    dd2::ProfRec *pr = dd2::prof_begin(DD_KERNEL_ADJOINT, st);
    int rc = launch_adj_kernel<GEOM, kNB>(a, 0, a.B / kNB, st);
    if (rc == DD_OK) rc = launch_adj_kernel<GEOM, 1>(a, a.B / kNB * kNB, a.B % kNB, st);
    dd2::prof_end(pr, st);
    return rc != DD_OK ? rc : launch_status();
}

// Forward-type operator into `out` (optionally minus `sub`).
int forward(int scan, int op, const dd_geom3d *g, const char *planb, const float *in, float *out,
            const float *sub, int B, int V, char *volx, char *volt, int *status, cudaStream_t st) {
    const int W = g->width, H = g->height, Dp = g->depth;
    const int pairs = B / kNB, odd = B % kNB;
    const long long nz = (long long)Dp * (pairs > 1 ? pairs : 1);
    const dim3 gl((unsigned)((W + 31) / 32), (unsigned)((H + 31) / 32), (unsigned)(nz < 65535 ? nz : 65535));
    const size_t done = (size_t)pairs * kNB * Dp;   // slices of the paired volumes
    dd2::ProfRec *pt = dd2::prof_begin(DD_KERNEL_TABLES, st);
    if (pairs) k_lines_of3<kNB><<<gl, 256, 0, st>>>(in, (float *)volx, (float *)volt, W, H, Dp, pairs, status);
    if (odd)
        k_lines_of3<1><<<gl, 256, 0, st>>>(in + done * W * H, (float *)volx + done * H * pad4(W),
                                           (float *)volt + done * W * pad4(H), W, H, Dp, 1, pairs ? nullptr : status);
    dd2::prof_end(pt, st);
    dd2::count_launches((pairs ? 1 : 0) + odd);
    const int s1 = launch_status();
    if (s1 != DD_OK) return s1;
    Fwd3Args a;
    a.status = status;
    a.g = *g;
    a.plan = planb;
    a.P = plan_layout(g, V);
    a.volx = (const float *)volx;
    a.volt = (const float *)volt;
    a.out = out;
    a.sub = sub;
    a.V = V;
    a.nrb = a.ncg = 0;
    a.b0 = 0;
    a.geom = geom_of(scan);
    a.family = op_family(op);
    dd2::ProfRec *pr = dd2::prof_begin(DD_KERNEL_FORWARD, st);
    int rc = launch_fwd_volumes<kNB>(a, 0, pairs, st);
    if (rc == DD_OK) rc = launch_fwd_volumes<1>(a, pairs * kNB, odd, st);
    dd2::prof_end(pr, st);
    return rc != DD_OK ? rc : launch_status();
}

// Adjoint-type operator: out = value, or out = base + scale * value.
int adjoint(int scan, int op, const dd_geom3d *g, const char *planb, const float *in, float *out,
            const float *basep, float scale, int B, int V, char *ss, int *status, cudaStream_t st) {
    Adj3Args a;
    a.status = status;
    a.g = *g;
    a.plan = planb;
    a.P = plan_layout(g, V);
    a.ss = (const float *)ss;
    a.out = out;
    a.base = basep;
    a.scale = scale;
    a.B = B;
    a.V = V;
    a.ntx = (g->width + kTile - 1) / kTile;
    a.b0 = 0;
    a.family = op_family(op);
    const int geom = geom_of(scan);
    if (geom == DD_GEOM3_CONE_FLAT) return launch_adj<DD_GEOM3_CONE_FLAT>(a, in, (float *)ss, st);
    if (geom == DD_GEOM3_CONE_ARC) return launch_adj<DD_GEOM3_CONE_ARC>(a, in, (float *)ss, st);
    return launch_adj<DD_GEOM3_SPIRAL>(a, in, (float *)ss, st);
}

}   // namespace dd3

using namespace dd3;

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
extern "C" int dd3d_validate(int scan, int op, const dd_geom3d *g, int batch, int num_view) {
    return validate(scan, op, g, batch, num_view);
}

extern "C" size_t dd3d_plan_bytes(int scan, const dd_geom3d *g, int num_view) {
    (void)scan;
    if (!g || num_view <= 0) return 0;
    return plan_layout(g, num_view).total;
}

extern "C" int dd3d_plan(int scan, const dd_geom3d *g, const float *angles, const float *source_pos, int num_view,
                         void *planp, size_t plan_bytes, dd_stream_t stream) {
    ddtrace::Range tr("dd3d_plan", scan, -1, true);
    const int st = validate(scan, DD_OP_PROJ, g, 1, num_view);
    if (st != DD_OK) return st;
    return plan(scan, g, angles, source_pos, num_view, planp, plan_bytes, (cudaStream_t)stream);
}

extern "C" size_t dd3d_apply_workspace_bytes(int scan, int op, const dd_geom3d *g, int batch, int num_view) {
    (void)scan;
    if (!g || batch <= 0 || num_view <= 0) return 0;
    const bool f = op_is_forward(op);
    return apply_layout(f, !f, g, batch, num_view).total;
}

extern "C" int dd3d_apply_planned(int scan, int op, const dd_geom3d *g, const void *planp, const float *in,
                                  float *out, int batch, int num_view, void *workspace, size_t workspace_bytes,
                                  dd_stream_t stream) {
    ddtrace::Range tr("dd3d_apply_planned", scan, op, true);
    const int st = validate(scan, op, g, batch, num_view);
    if (st != DD_OK) return st;
    if (!planp || !in || !out) return DD_ERR_INVALID_ARG;
    const bool f = op_is_forward(op);
    const ApplyLayout A = apply_layout(f, !f, g, batch, num_view);
    if (!workspace || workspace_bytes < A.total) return DD_ERR_WORKSPACE;
    char *wb = ws_base(workspace);
    cudaStream_t s = (cudaStream_t)stream;
    int *status = (int *)(wb + A.status);
    if (f) return forward(scan, op, g, (const char *)planp, in, out, nullptr, batch, num_view, wb + A.volx, wb + A.volt, status, s);
    return adjoint(scan, op, g, (const char *)planp, in, out, nullptr, 0.0f, batch, num_view, wb + A.ss, status, s);
}

extern "C" size_t dd3d_workspace_bytes(int scan, int op, const dd_geom3d *g, int batch, int num_view) {
    if (!g || batch <= 0 || num_view <= 0) return 0;
    return dd3d_plan_bytes(scan, g, num_view) + dd3d_apply_workspace_bytes(scan, op, g, batch, num_view);
}

extern "C" int dd3d_apply(int scan, int op, const dd_geom3d *g, const float *in, float *out, const float *angles,
                          const float *source_pos, int batch, int num_view, void *workspace,
                          size_t workspace_bytes, dd_stream_t stream) {
    ddtrace::Range tr("dd3d_apply", scan, op, true);
    const int st = validate(scan, op, g, batch, num_view);
    if (st != DD_OK) return st;
    if (!in || !out || !angles || (scan == DD_SCAN_SPIRAL && !source_pos)) return DD_ERR_INVALID_ARG;
    const size_t pb = dd3d_plan_bytes(scan, g, num_view);
    if (!workspace || workspace_bytes < dd3d_workspace_bytes(scan, op, g, batch, num_view)) return DD_ERR_WORKSPACE;
    char *wb = ws_base(workspace);
    const int s1 = plan(scan, g, angles, source_pos, num_view, wb, pb, (cudaStream_t)stream);
    if (s1 != DD_OK) return s1;
    return dd3d_apply_planned(scan, op, g, wb, in, out, batch, num_view, wb + pb, workspace_bytes - pb, stream);
}

extern "C" size_t dd3d_dc_workspace_bytes(int scan, const dd_geom3d *g, int batch, int num_view) {
    (void)scan;
    if (!g || batch <= 0 || num_view <= 0) return 0;
    return apply_layout(true, true, g, batch, num_view).total;
}

extern "C" int dd3d_dc_step(int scan, const dd_geom3d *g, const void *planp, float *x, const float *y, float *resid,
                            float eta, int batch, int num_view, void *workspace, size_t workspace_bytes,
                            dd_stream_t stream) {
    ddtrace::Range tr("dd3d_dc_step", scan, -1, true);
    const int st = validate(scan, DD_OP_PROJ, g, batch, num_view);
    if (st != DD_OK) return st;
    if (!planp || !x || !y || !resid) return DD_ERR_INVALID_ARG;
    const ApplyLayout A = apply_layout(true, true, g, batch, num_view);
    if (!workspace || workspace_bytes < A.total) return DD_ERR_WORKSPACE;
    char *wb = ws_base(workspace);
    cudaStream_t s = (cudaStream_t)stream;
    const char *pb = (const char *)planp;
    int *status = (int *)(wb + A.status);
    const int s1 = forward(scan, DD_OP_PROJ, g, pb, x, resid, y, batch, num_view, wb + A.volx, wb + A.volt, status, s);
    if (s1 != DD_OK) return s1;
    return adjoint(scan, DD_OP_PROJ_T, g, pb, resid, x, x, -eta, batch, num_view, wb + A.ss, status + 1, s);
}

extern "C" int dd3d_status(int scan, int op, const dd_geom3d *g, int batch, int num_view, const void *workspace,
                           int *status) {
    if (validate(scan, op, g, batch, num_view) != DD_OK || !workspace || !status) return DD_ERR_INVALID_ARG;
    const bool f = op_is_forward(op);
    const size_t off = dd3d_plan_bytes(scan, g, num_view) + apply_layout(f, !f, g, batch, num_view).status;
    if (cudaMemcpy(status, ws_base(workspace) + off, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
        return DD_ERR_LAUNCH;
    return DD_OK;
}

extern "C" int dd3d_planned_status(int op, const dd_geom3d *g, int batch, int num_view, const void *workspace,
                                   int *status) {
    if (!g || batch <= 0 || num_view <= 0 || !workspace || !status) return DD_ERR_INVALID_ARG;
    const bool f = op_is_forward(op);
    const size_t off = apply_layout(f, !f, g, batch, num_view).status;
    if (cudaMemcpy(status, ws_base(workspace) + off, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
        return DD_ERR_LAUNCH;
    return DD_OK;
}

int dd3_set_sink(int *sink) { return dd_set_status_sink_tu(sink); }

// named entries (RadonTorch.cpp:1395-1414)
#define DD_NAMED3(name, scan, op)                                                                          \
    extern "C" int dd_##name(const dd_geom3d *g, const float *in, float *out, const float *angles,           \
                             const float *source_pos, int batch, int num_view, void *workspace,             \
                             size_t workspace_bytes, dd_stream_t stream) {                                  \
        return dd3d_apply(scan, op, g, in, out, angles, source_pos, batch, num_view, workspace,            \
                          workspace_bytes, stream);                                                         \
    }
DD_NAMED3(ProjConeFlatDis3d, DD_SCAN_CONE_FLAT, DD_OP_PROJ)
DD_NAMED3(ProjTransConeFlatDis3d, DD_SCAN_CONE_FLAT, DD_OP_PROJ_T)
DD_NAMED3(BackProjConeFlatDis3d, DD_SCAN_CONE_FLAT, DD_OP_BPROJ)
DD_NAMED3(BackProjTransConeFlatDis3d, DD_SCAN_CONE_FLAT, DD_OP_BPROJ_T)
DD_NAMED3(BackProjWeightedConeFlatDis3d, DD_SCAN_CONE_FLAT, DD_OP_BPROJ_W)
DD_NAMED3(BackProjTransWeightedConeFlatDis3d, DD_SCAN_CONE_FLAT, DD_OP_BPROJ_TW)
DD_NAMED3(ProjConeArcDis3d, DD_SCAN_CONE_ARC, DD_OP_PROJ)
DD_NAMED3(ProjTransConeArcDis3d, DD_SCAN_CONE_ARC, DD_OP_PROJ_T)
DD_NAMED3(BackProjConeArcDis3d, DD_SCAN_CONE_ARC, DD_OP_BPROJ)
DD_NAMED3(BackProjTransConeArcDis3d, DD_SCAN_CONE_ARC, DD_OP_BPROJ_T)
DD_NAMED3(BackProjWeightedConeArcDis3d, DD_SCAN_CONE_ARC, DD_OP_BPROJ_W)
DD_NAMED3(BackProjTransWeightedConeArcDis3d, DD_SCAN_CONE_ARC, DD_OP_BPROJ_TW)
DD_NAMED3(ProjSpiralDis3d, DD_SCAN_SPIRAL, DD_OP_PROJ)
DD_NAMED3(ProjTransSpiralDis3d, DD_SCAN_SPIRAL, DD_OP_PROJ_T)
DD_NAMED3(BackProjSpiralDis3d, DD_SCAN_SPIRAL, DD_OP_BPROJ)
DD_NAMED3(BackProjTransSpiralDis3d, DD_SCAN_SPIRAL, DD_OP_BPROJ_T)
DD_NAMED3(BackProjWeightedSpiralDis3d, DD_SCAN_SPIRAL, DD_OP_BPROJ_W)
DD_NAMED3(BackProjTransWeightedSpiralDis3d, DD_SCAN_SPIRAL, DD_OP_BPROJ_TW)
#undef DD_NAMED3
