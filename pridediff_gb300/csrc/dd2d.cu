// GB300 (sm_103a) 2-D distance-driven projector: parallel, fan-flat, fan-arc.
//
// Replaces the 16 2-D operators of deeprecon's radontorch extension
// (RadonTorch.cpp:17-568; kernels deeprecon/cuda/dis2d/*.cu, CPU path
// deeprecon/cpu/dis2d/*.cpp).  Results follow the reference CPU path, which is
// the parity target.
//
// Algorithm (integral form of the DD merge walk).  For one view and one
// walked image line, deeprecon merges the sorted pixel boundaries b_i and
// detector boundaries d_k on a projection axis and weights every overlap
// segment.  The same sums are differences of integrals:
//   forward (detector gathers):  bin_k  += F(d_{k+1}) - F(d_k),
//                                F(u) = integral of the pixel function to u;
//   adjoint (pixel gathers):     pix_i  += H(b_i) - H(b_{i-1}),
//                                H(u) = integral of the detector function.
// H is evaluated from a per-view prefix table of the detector row, staged in
// shared memory by TMA bulk copies: branch-free interpolations, so a warp
// processes 32 adjacent boundaries in lock step and neighbouring lanes
// exchange values with one shuffle.  The adjoint is a gather: no atomics,
// deterministic.  The forward's difference of integrals is the sum of a
// bin's overlaps with the line's pixels, at most a few: they are taken from a
// table of the line's boundaries, once for all the slices of a group
// (dd2d_fwd.cuh).  One or two slices of an arc fan take F from a per-line
// prefix table as well (dd2d_prefix.cuh).
//
// The pixel boundaries are deeprecon's drifted FP32 sequence
// (`Point1Proj += PixInterval`), represented exactly by per-line binade
// pieces (dd_geom.cuh); an integral over drifted pixels is then
//   K_p + dl_p * S_j + r * x_j
// with a per-piece constant K_p computed once per line by a warp scan.
#include <cuda_runtime.h>

#include <algorithm>
#include <stdint.h>
#include <string.h>

#include "dd2d_fwd.cuh"
#include "dd2d_prefix.cuh"
#include "dd_trace.h"

namespace dd2 {
// ---------------------------------------------------------------------------
// Plan kernels
// ---------------------------------------------------------------------------
__global__ void k_views(int geom, dd_geom2d g, const float *__restrict__ angles, int V,
                        DdView2 *__restrict__ views, float *__restrict__ ang,
                        float *__restrict__ dp, float *__restrict__ bcoef) {
    const int v = blockIdx.x;
    if (v >= V) return;
    const float view = angles[v];
    DdView2 vw;
    dd_view2_scalars(geom, &g, view, &vw);
    if (threadIdx.x == 0) {
        views[v] = vw;
        ang[v] = view;
    }
    if (geom == DD_GEOM_PARA) return;
    const int D = g.num_det;
    float *dpv = dp + (size_t)v * (D + 1);
    for (int k = threadIdx.x; k <= D; k += blockDim.x) dpv[k] = dd_view2_boundary(geom, &g, view, &vw, k);
    __syncthreads();
    float *bc = bcoef + (size_t)v * (D + 1);
    for (int k = threadIdx.x; k < D; k += blockDim.x) bc[k] = dd_view2_bcoef(&g, &vw, dpv[k], dpv[k + 1]);
}

__global__ void k_lines(int geom, dd_geom2d g, const float *__restrict__ angles, int V, int nl,
                        const DdView2 *__restrict__ views, const float *__restrict__ dp,
                        DdLine *__restrict__ lines, DdLine *__restrict__ dlines) {
    const int v = blockIdx.y;
    const int line = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const DdView2 vw = views[v];
    const int nline = vw.xb ? g.height : g.width;
    if (line >= nline) return;
    const size_t r = (size_t)v * nl + line;
    dd_line2_setup(geom, &g, angles[v], &vw, dp + (size_t)v * (g.num_det + 1), line, lines + r,
                   dlines ? dlines + r : nullptr);
}

// ---------------------------------------------------------------------------
// Forward: planes of rows and columns, and the single-geometry launch
// ---------------------------------------------------------------------------
// Planes of P slices of a stack of B images: the rows (lines of the views
// that walk rows) and the columns from the bottom row up (dd2d_fwd.cuh).
template <int P>
__global__ void __launch_bounds__(256)
k_planes(const float *__restrict__ img, int B, int H, int W, float *__restrict__ rows, float *__restrict__ cols,
         size_t rplane, size_t cplane, int *__restrict__ clear) {
    __shared__ float t[32][33 * P];
    if (clear && threadIdx.x == 0 && blockIdx.x + blockIdx.y + blockIdx.z == 0) *clear = 0;   // the call's status word
    const int q = blockIdx.z;
    plane_tile<P>(img + (size_t)q * P * H * W, min(P, B - q * P), W, H, blockIdx.x * 32, blockIdx.y * 32,
                  rows + q * rplane, cols + q * cplane, t);
}

// Detector tables for the adjoint: per (image, view) G_k and g_k over the
// sorted bins.  Fan: G_k = sum_{m<k} g_m (d_{m+1} - d_m) (exact widths);
// parallel: unit prefix (the drifted widths enter through the line pieces).
// mode 0: g = s * bcoef (ProjTrans), mode 1: g = s (BackProj family).
__global__ void k_dettab(int geom, int mode, const float *__restrict__ sino, int B, int V, int D,
                         const DdView2 *__restrict__ views, const float *__restrict__ dp,
                         const float *__restrict__ bcoef, float para_coef_x, float para_coef_y,
                         float2 *__restrict__ tab, int *__restrict__ clear) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (blockIdx.x + threadIdx.x == 0) *clear = 0;   // the call's status word
    if (warp >= B * V) return;
    const int b = warp / V, v = warp - b * V;
    const DdView2 vw = views[v];
    const float *s = sino + ((size_t)b * V + v) * D;
    const float *dpv = dp + (size_t)v * (D + 1);
    const float *bc = bcoef + (size_t)v * (D + 1);
    const float pc = vw.xb ? para_coef_x : para_coef_y;
    warp_prefix_table(D, tab + (size_t)warp * rs_entries(D), lane, [&](int k, float *g, float *w) {
        const float sv = s[vw.flip ? D - 1 - k : k];
        if (geom == DD_GEOM_PARA) {
            *g = (mode == 0) ? sv * pc : sv;
            *w = 1.0f;
        } else {
            *g = (mode == 0) ? sv * bc[k] : sv;
            *w = dpv[k + 1] - dpv[k];
        }
    });
}

// Single-geometry forward: one item per cluster.  blockIdx.x = view * cluster
// size + rank, blockIdx.y = group of NB slices.  3 CTAs per SM (56 registers)
// up to 24 sums a thread.
template <int KIND, int NPASS, int NB, bool WIDE>
__global__ void __launch_bounds__(fwd_threads(NB), NPASS * NB <= 24 ? 3 : 2)
k_fwd(dd_geom2d g, int geom, int op, int B, int V, int nl, const DdView2 *__restrict__ views,
      const float *__restrict__ dp, const float *__restrict__ bcoef, const DdLine *__restrict__ lines,
      const DdLine *__restrict__ dlines, const float *__restrict__ rows, const float *__restrict__ cols,
      size_t rplane, size_t cplane, float *__restrict__ out, const float *__restrict__ sub, int cl, int sh, int ks,
      int *__restrict__ status) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ FwdState S;
    // (a constant where there is no choice: the stages' indices are then cheaper)
    const FwdLay L = fwd_lay(KIND, g.num_det, g.num_det << sh, max(g.width, g.height), NB, cl,
                             stages(NB) > prods(NB) ? ks : stages(NB));
    fwd_init<KIND, NB>(smem, L, S);
    constexpr int planes = NB / plane_slices(NB);
    FwdItem it;
    it.v = blockIdx.x / cl;
    it.b0 = blockIdx.y * NB;
    it.nb = min(NB, B - it.b0);
    it.V = V;
    it.nl = nl;
    it.sh = sh;
    it.views = views;
    it.dp = dp;
    it.bcoef = bcoef;
    it.lines = lines;
    it.dlines = dlines;
    it.rows = rows + (size_t)blockIdx.y * planes * rplane;
    it.cols = cols + (size_t)blockIdx.y * planes * cplane;
    it.rplane = rplane;
    it.cplane = cplane;
    it.out = out;
    it.sub = sub;
    uint32_t step = 0, nr = 0;
    if (!fwd_item<KIND, NPASS, NB, WIDE>(g, geom, op, it, smem, L, S, step, nr) && threadIdx.x == 0) dd_report_timeout(status);
}

// Plan time: the views that walk image rows and those that walk columns, each
// in view order.  One warp: ballots rank the views.
__global__ void __launch_bounds__(32)
k_axis_views(int V, const DdView2 *__restrict__ views, int *__restrict__ axisv) {
    const int lane = threadIdx.x;
    const unsigned below = (1u << lane) - 1u;
    int nr = 0, nc = 0;
    for (int v0 = 0; v0 < V; v0 += 32) {
        const int v = v0 + lane;
        const bool in = v < V;
        const bool xb = in && views[v].xb;
        const unsigned mr = __ballot_sync(0xffffffffu, xb), mc = __ballot_sync(0xffffffffu, in && !xb);
        if (xb) axisv[2 + nr + __popc(mr & below)] = v;
        else if (in) axisv[2 + V + nc + __popc(mc & below)] = v;
        nr += __popc(mr);
        nc += __popc(mc);
    }
    if (lane == 0) {
        axisv[0] = nr;
        axisv[1] = nc;
    }
}

// Single-geometry parallel-beam adjoint launch: grid (lines * cluster, image groups).
template <int OPK, int NQ>   // OPK: 0 ProjTrans, 1 BackProj; NQ: pixels a thread without clusters (0: clusters)
__global__ void __launch_bounds__(kThreads)
k_adj_para(dd_geom2d g, int B, int V, int nl, int axis, const int *__restrict__ axisv,
           const DdLine *__restrict__ lines, const DdLine *__restrict__ dlines,
           const float2 *__restrict__ dtab, float *__restrict__ out, const float *__restrict__ base,
           float scale, int *__restrict__ status) {
    extern __shared__ __align__(128) unsigned char smem[];
    AdjItem it = {};
    it.c0 = blockIdx.x / (NQ > 0 ? 1 : kAdjCluster);
    it.r0 = axis;
    it.b0 = blockIdx.y * kBI;
    it.nb = min(kBI, B - it.b0);
    it.V = V;
    it.nl = nl;
    it.lines = lines;
    it.dlines = dlines;
    it.axisv = axisv;
    it.dtab = dtab;
    it.out = out;
    it.base = base;
    it.scale = scale;
    const ParaSmem S = para_smem(g.num_det, axis ? g.width : g.height, min(kBI, B));
    if (!adj_para_line<OPK, NQ>(g, it, smem, S) && threadIdx.x == 0) dd_report_timeout(status);
}

// Adjoint map of fan beams (plan time): one CTA per (tile, view) fills the
// tile's block.  For each of the tile's walked lines and boundary indices
// b = e - 1 (e from map_first()): the detector bin k and offset u - d_k of the
// clamped boundary value u, exactly as the pixel-gather adjoint needs them
// (k = -1 where the walk does not reach b; boundary i0 - 1 is the walk
// start); then the lines' DD-BP scales.
template <int GEOM>
__global__ void __launch_bounds__(128)
k_amap(dd_geom2d g, int nl, const DdView2 *__restrict__ views, const float *__restrict__ angles,
       const float *__restrict__ dp, const DdLine *__restrict__ lines, unsigned char *__restrict__ amap) {
    const int t = blockIdx.x, v = blockIdx.y;
    const int c0 = (t % tiles_x(&g)) * kTile, r0 = (t / tiles_x(&g)) * kTile;
    const int ms = map_stride(&g), D = g.num_det;
    const DdView2 vw = views[v];
    const int nline = vw.xb ? g.height : g.width;
    const int l0 = vw.xb ? r0 : c0, elo = map_first(&g, vw.xb, c0, r0);
    int2 *ent = reinterpret_cast<int2 *>(amap + ((size_t)v * tiles_n(&g) + t) * kMapBlkBytes);
    float *alpha = reinterpret_cast<float *>(ent + kTile * kMapE);
    const float *dpv = dp + (size_t)v * (D + 1);
    const float ang = angles[v];
    for (int i = threadIdx.x; i < kTile * kMapE; i += 128) {
        const int li = i / kMapE, e = elo + (i - li * kMapE), line = l0 + li;
        int2 val = make_int2(-1, 0);
        if (line < nline && e < ms) {
            const DdLine &L = lines[(size_t)v * nl + line];
            const int b = e - 1, i0 = L.h.i0, nend = L.h.nend;
            if (L.h.npiece > 0 && b >= i0 - 1 && b < nend) {
                const float bound0 = L.h.bound0;
                const float u =
                    (b == i0 - 1) ? bound0 : dd_boundary(&L, b, L.p[0].Q + (float)(b - L.p[0].gb) * L.p[0].dl);
                const float uu = fminf(fmaxf(u, bound0), dpv[D]);
                float dk;
                const int k = fan_bin(GEOM, g, vw, ang, dpv, uu, L.h.idet0, &dk);
                val = make_int2(k, __float_as_int(uu - dk));
            }
        }
        ent[i] = val;
    }
    if (threadIdx.x < kTile) {
        const int line = l0 + threadIdx.x;
        alpha[threadIdx.x] = line < nline ? lines[(size_t)v * nl + line].h.alpha : 0.0f;
    }
}

// Detector-table slice staged per (view, 32x32 tile) by the fan-beam adjoint
// (plan time): the tile's bin range (tile_bin_range) rounded to an even first
// bin and an even count (16-byte bulk copies), or count 0 when wider than the
// staging buffer.  One thread per (view, tile).
template <int GEOM>
__global__ void __launch_bounds__(128)
k_trange(dd_geom2d g, int V, const DdView2 *__restrict__ views, const float *__restrict__ angles,
         int2 *__restrict__ trange) {
    const int nt = tiles_n(&g);
    const int i = blockIdx.x * 128 + threadIdx.x;
    if (i >= V * nt) return;
    const int v = i / nt, t = i - v * nt;
    const int c0 = (t % tiles_x(&g)) * kTile, r0 = (t / tiles_x(&g)) * kTile;
    int kmin, kmax;
    tile_bin_range(GEOM, g, views[v], angles[v], c0, r0, &kmin, &kmax);
    const int rsd = rs_entries(g.num_det);
    const int kb = kmin & ~1;
    int kn = (kmax - kb + 2) & ~1;
    if (kb + kn > rsd) kn = rsd - kb;
    if (kn > kStage || kn <= 0) kn = 0;
    trange[i] = make_int2(kb, kn | (views[v].xb ? 1 << 16 : 0));   // the view's axis in bit 16
}

// Single-geometry fan-beam adjoint launch: grid (tiles x * image groups *
// cluster, tiles y); 4 CTAs per SM (64 registers), as the persistent adjoint.
template <int GEOM, int OPK, int NB>
__global__ void __cluster_dims__(kAdjCluster, 1, 1) __launch_bounds__(kThreads, 4)
k_adj(dd_geom2d g, int B, int V, const DdView2 *__restrict__ views, const unsigned char *__restrict__ amap,
      const int2 *__restrict__ trange, const int *__restrict__ axisv, const float2 *__restrict__ dtab,
      float *__restrict__ out, const float *__restrict__ base, float scale, int *__restrict__ status) {
    extern __shared__ __align__(128) unsigned char smem[];
    const AdjSmem SL = adj_smem();
    init_bars(reinterpret_cast<uint64_t *>(smem + SL.bar), kAdjBufs);
    DdPhases ph;
    AdjItem it = {};
    // the image groups of a tile are adjacent in launch order: they run at the
    // same time, walk the views in step and read each view's map block of the
    // tile once from DRAM between them (the others hit L2)
    const int ngroups = (B + NB - 1) / NB, at = blockIdx.x / kAdjCluster;
    it.c0 = (at / ngroups) * kTile;
    it.r0 = blockIdx.y * kTile;
    it.b0 = (at % ngroups) * NB;
    it.nb = min(NB, B - it.b0);
    it.V = V;
    it.views = views;
    it.amap = amap;
    it.trange = trange;
    it.axisv = axisv;
    it.dtab = dtab;
    it.out = out;
    it.base = base;
    it.scale = scale;
    if (!adj_tile_map<GEOM, OPK, NB>(g, it, smem, ph) && threadIdx.x == 0) dd_report_timeout(status);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
int geom_of(int scan) {
    return scan == DD_SCAN_PARA ? DD_GEOM_PARA : (scan == DD_SCAN_FLAT ? DD_GEOM_FLAT : DD_GEOM_ARC);
}

int validate(int scan, int op, const dd_geom2d *g, int B, int V) {
    if (!g) return DD_ERR_INVALID_ARG;
    if (scan < DD_SCAN_PARA || scan > DD_SCAN_ARC) return DD_ERR_INVALID_ARG;
    if (op < DD_OP_PROJ || op > DD_OP_BPROJ_TW) return DD_ERR_INVALID_ARG;
    if (scan == DD_SCAN_PARA && (op == DD_OP_BPROJ_W || op == DD_OP_BPROJ_TW)) return DD_ERR_UNSUPPORTED;
    if (g->width <= 0 || g->height <= 0 || g->num_det <= 0 || B <= 0 || V <= 0) return DD_ERR_INVALID_ARG;
    const float f[] = {g->pix_x, g->pix_y, g->det_size, g->iso_source, g->source_detector,
                       g->pix_xshift, g->pix_yshift, g->bin_shift};
    for (float x : f)
        if (!(x == x) || x - x != 0.0f) return DD_ERR_INVALID_ARG;   // NaN / inf
    if (!(g->pix_x > 0 && g->pix_y > 0 && g->det_size > 0)) return DD_ERR_INVALID_ARG;
    if (scan != DD_SCAN_PARA && !(g->iso_source > 0 && g->source_detector > 0)) return DD_ERR_INVALID_ARG;
    const long long lim = (1LL << 31) - 1;
    if ((long long)g->width * g->height * B > lim) return DD_ERR_SIZE_OVERFLOW;
    if ((long long)V * g->num_det * B > lim) return DD_ERR_SIZE_OVERFLOW;
    if (g->width > 4096 || g->height > 4096) return DD_ERR_SIZE_OVERFLOW;
    if (g->num_det > 8 * kWarps * kBinsPerWarp) return DD_ERR_SIZE_OVERFLOW;
    return DD_OK;
}

int launch_status() {
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? DD_OK : DD_ERR_LAUNCH;
}

// ---------------------------------------------------------------------------
// Launch accounting and optional per-kernel event timing (benchmarks only;
// never enabled during graph capture)
// ---------------------------------------------------------------------------
static unsigned long long g_launches = 0;
static int g_prof = 0;
struct ProfRec {
    cudaEvent_t a, b;
    int kind;
};
static ProfRec g_prof_rec[8192];
static int g_prof_used = 0;
static int g_prof_created = 0;

ProfRec *prof_begin(int kind, cudaStream_t st) {
    if (!g_prof || g_prof_used >= 8192) return nullptr;
    ProfRec *r = &g_prof_rec[g_prof_used];
    if (g_prof_used >= g_prof_created) {
        if (cudaEventCreate(&r->a) != cudaSuccess || cudaEventCreate(&r->b) != cudaSuccess) return nullptr;
        g_prof_created++;
    }
    g_prof_used++;
    r->kind = kind;
    cudaEventRecord(r->a, st);
    return r;
}
void prof_end(ProfRec *r, cudaStream_t st) {
    if (r) cudaEventRecord(r->b, st);
}

void count_launches(int n) { g_launches += (unsigned long long)n; }

int plan(int scan, const dd_geom2d *g, const float *angles, int V, void *planp, size_t bytes,
         cudaStream_t st, bool with_map) {
    const PlanLayout P = plan_layout(scan, g, V, with_map);
    if (!planp || bytes < P.total) return DD_ERR_WORKSPACE;
    if (!angles) return DD_ERR_INVALID_ARG;
    char *base = (char *)planp;
    const int geom = geom_of(scan);
    DdView2 *views = (DdView2 *)(base + P.views);
    float *dp = (float *)(base + P.dp);
    float *bc = (float *)(base + P.bcoef);
    DdLine *lines = (DdLine *)(base + P.lines);
    DdLine *dlines = scan == DD_SCAN_PARA ? (DdLine *)(base + P.dlines) : nullptr;
    ProfRec *pr = prof_begin(DD_KERNEL_PLAN, st);
    k_views<<<V, 256, 0, st>>>(geom, *g, angles, V, views, (float *)(base + P.ang), dp, bc);
    if (geom == DD_GEOM_PARA || with_map) {
        k_axis_views<<<1, 32, 0, st>>>(V, views, (int *)(base + P.axisv));
        g_launches++;
    }
    dim3 gl((P.nl + 63) / 64, V);
    k_lines<<<gl, 64, 0, st>>>(geom, *g, angles, V, P.nl, views, dp, lines, dlines);
    int n = 2;
    if (geom != DD_GEOM_PARA && with_map) {
        const dim3 gm((unsigned)tiles_n(g), (unsigned)V);
        const float *ang = (const float *)(base + P.ang);
        unsigned char *amap = (unsigned char *)(base + P.amap);
        int2 *trange = (int2 *)(base + P.trange);
        const int nt = (V * tiles_n(g) + 127) / 128;
        if (geom == DD_GEOM_FLAT) {
            k_amap<DD_GEOM_FLAT><<<gm, 128, 0, st>>>(*g, P.nl, views, ang, dp, lines, amap);
            k_trange<DD_GEOM_FLAT><<<nt, 128, 0, st>>>(*g, V, views, ang, trange);
        } else {
            k_amap<DD_GEOM_ARC><<<gm, 128, 0, st>>>(*g, P.nl, views, ang, dp, lines, amap);
            k_trange<DD_GEOM_ARC><<<nt, 128, 0, st>>>(*g, V, views, ang, trange);
        }
        n += 2;
    }
    prof_end(pr, st);
    g_launches += n;
    return launch_status();
}

// Largest dynamic shared memory a CTA may opt in to on this device.
int max_smem_optin() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&n, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess || n <= 0)
            n = 227 * 1024;   // no device to ask (host-side checks): the sm_103a figure
    }
    return n;
}

int sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
            n = 1;
    }
    return n;
}

// The forward CTA shape a tune asks for (slices per CTA, CTAs per view's
// cluster), with the defaults where it asks for none, and 1 slice where lines
// are too long for 4.
static void fwd_shape(int geom, const dd_geom2d *g, const dd_tune2d *tune, int *bi, int *cl) {
    *bi = (tune && (tune->fwd_slices == 1 || tune->fwd_slices == 4)) ? tune->fwd_slices : 4;
    *cl = (tune && (tune->fwd_cluster == 1 || tune->fwd_cluster == 2)) ? tune->fwd_cluster : 2;
    if (*bi == 4 && four_slice_bytes(geom == DD_GEOM_PARA, g->num_det, std::max(g->width, g->height), *cl) > max_smem_optin())
        *bi = 1;
}

struct FwdCall {
    const dd_geom2d *g;
    int geom, op, V, nl, cl, sh;
    const DdView2 *views;
    const float *dp, *bcoef;
    const DdLine *lines, *dlines;
    const float *sub;
    int *status;
    bool first;   // the call's first launch, which clears its status word
    cudaStream_t st;
};

// `n` slices in groups of NB: their planes, and the groups' items.
template <int KIND, int NPASS, int NB, bool WIDE>
static int launch_fwd_group(const FwdCall &c, const float *in, int n, float *rows, float *cols, float *out,
                            const float *sub) {
    constexpr int P = plane_slices(NB);
    const int W = c.g->width, H = c.g->height, groups = (n + NB - 1) / NB;
    const size_t rplane = plane_bytes(H, W, P) / sizeof(float), cplane = plane_bytes(W, H, P) / sizeof(float);
    const int planes = groups * (NB / P);
    if (planes > 65535) return DD_ERR_SIZE_OVERFLOW;
    ProfRec *pt = prof_begin(DD_KERNEL_TABLES, c.st);
    k_planes<P><<<dim3((unsigned)((W + 31) / 32), (unsigned)((H + 31) / 32), (unsigned)planes), 256, 0, c.st>>>(
        in, n, H, W, rows, cols, rplane, cplane, c.first ? c.status : nullptr);
    prof_end(pt, c.st);
    const FwdLay L = fwd_lay(KIND, c.g->num_det, c.g->num_det << c.sh, std::max(W, H), NB, c.cl);
    auto kern = k_fwd<KIND, NPASS, NB, WIDE>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L.total) != cudaSuccess)
        return DD_ERR_LAUNCH;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)c.cl;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(c.V * c.cl), (unsigned)groups);
    cfg.blockDim = dim3(fwd_threads(NB));
    cfg.dynamicSmemBytes = (size_t)L.total;
    cfg.stream = c.st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    ProfRec *pr = prof_begin(DD_KERNEL_FORWARD, c.st);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, *c.g, c.geom, c.op, n, c.V, c.nl, c.views, c.dp, c.bcoef, c.lines,
                                             c.dlines, (const float *)rows, (const float *)cols, rplane, cplane, out, sub,
                                             c.cl, c.sh, L.ks, c.status);
    prof_end(pr, c.st);
    g_launches += 2;
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return DD_ERR_LAUNCH;
    }
    return launch_status();
}

template <int KIND, int NB>
static int launch_fwd_passes(const FwdCall &c, const float *in, int n, float *rows, float *cols, float *out,
                             const float *sub) {
    if (c.sh > 0)   // wide bins: at most two passes
        return c.g->num_det << c.sh <= kBins ? launch_fwd_group<KIND, 1, NB, true>(c, in, n, rows, cols, out, sub)
                                             : launch_fwd_group<KIND, 2, NB, true>(c, in, n, rows, cols, out, sub);
    switch (pass_class(c.g->num_det)) {
    case 1: return launch_fwd_group<KIND, 1, NB, false>(c, in, n, rows, cols, out, sub);
    case 2: return launch_fwd_group<KIND, 2, NB, false>(c, in, n, rows, cols, out, sub);
    case 3: return launch_fwd_group<KIND, 3, NB, false>(c, in, n, rows, cols, out, sub);
    case 4: return launch_fwd_group<KIND, 4, NB, false>(c, in, n, rows, cols, out, sub);
    default: return launch_fwd_group<KIND, 8, (NB > 4 ? 4 : NB), false>(c, in, n, rows, cols, out, sub);   // never 8 slices
    }
}

// Groups of 8 slices of the weighted transpose without its table.
static int launch_fwd_each(const FwdCall &c, const float *in, int n, float *rows, float *cols, float *out, const float *sub) {
    switch (pass_class(c.g->num_det)) {
    case 1: return launch_fwd_group<kFanWeightedEach, 1, 8, false>(c, in, n, rows, cols, out, sub);
    case 2: return launch_fwd_group<kFanWeightedEach, 2, 8, false>(c, in, n, rows, cols, out, sub);
    case 3: return launch_fwd_group<kFanWeightedEach, 3, 8, false>(c, in, n, rows, cols, out, sub);
    default: return launch_fwd_group<kFanWeightedEach, 4, 8, false>(c, in, n, rows, cols, out, sub);
    }
}

// One or two slices of an arc fan (dd2d_prefix.cuh).
template <int NPASS, int BI>
static int launch_prefix_as(const FwdCall &c, int B, const float *in, float2 *tx, float2 *ty, float *out) {
    const int W = c.g->width, H = c.g->height;
    ProfRec *pt = prof_begin(DD_KERNEL_TABLES, c.st);
    k_tab_rows<<<(unsigned)(((size_t)B * H * 32 + 255) / 256), 256, 0, c.st>>>(in, B, H, W, tx, c.status);
    k_tab_cols<<<B * ((W + 31) / 32), 32 * kColChunks, 0, c.st>>>(in, B, H, W, ty);
    prof_end(pt, c.st);
    const PrefixSmem S = prefix_smem(c.g->num_det, rs_entries(std::max(W, H)), BI);
    auto kern = k_fwd_prefix<NPASS, BI>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S.total) != cudaSuccess)
        return DD_ERR_LAUNCH;
    ProfRec *pr = prof_begin(DD_KERNEL_FORWARD, c.st);
    kern<<<(unsigned)c.V * 2, kThreads, S.total, c.st>>>(*c.g, B, c.V, c.nl, c.views, c.dp, c.bcoef, c.lines, tx, ty,
                                                         out, c.sub, c.status);
    prof_end(pr, c.st);
    g_launches += 3;
    return launch_status();
}
template <int BI>
static int launch_prefix(const FwdCall &c, int B, const float *in, float2 *tx, float2 *ty, float *out) {
    switch (prefix_passes(c.g->num_det)) {
    case 1: return launch_prefix_as<1, BI>(c, B, in, tx, ty, out);
    case 2: return launch_prefix_as<2, BI>(c, B, in, tx, ty, out);
    case 3: return launch_prefix_as<3, BI>(c, B, in, tx, ty, out);
    case 4: return launch_prefix_as<4, BI>(c, B, in, tx, ty, out);
    default: return launch_prefix_as<8, BI>(c, B, in, tx, ty, out);
    }
}

// Slices per CTA: 8 share a line's overlaps best; groups of 8, then 4 (of
// which one may be empty), 2 or 1 for the rest.  5 to 7 left over take one
// group of 8: about the time of two smaller ones.  No 8 where the stages of
// three lines would leave room for one CTA per SM only (lines of more than
// about 1,000 pixels) or the detector needs 8 passes (the sums' registers).
// 4 or 2 where they fit; one slice always does (4,096 pixels, 1,984 cells).
template <int KIND>
static int launch_fwd(FwdCall c, bool single, int B, const float *in, char *rows, char *cols, float *out) {
    const int W = c.g->width, H = c.g->height, D = c.g->num_det, npix = std::max(W, H), lanes = D << c.sh;
    if ((long long)c.V * c.cl > 0x7FFFFFFFLL) return DD_ERR_SIZE_OVERFLOW;
    const size_t image = (size_t)W * H, sino = (size_t)c.V * D;
    int big = 1;
    if (!single) {
        const int limit = max_smem_optin();
        big = pass_class(lanes) <= 4 && fwd_lay(KIND, D, lanes, npix, 8, c.cl).total <= limit / 2 ? 8
              : fwd_fits(KIND, D, lanes, npix, 4, c.cl, limit)                                ? 4
              : fwd_fits(KIND, D, lanes, npix, 2, c.cl, limit)                                ? 2
                                                                                                : 1;
    }
    // 8 slices fit, but not beside the weights of the line's pixels
    const bool each = KIND == kFanWeighted && !single && big < 8 && c.sh == 0 && pass_class(D) <= 4 &&
                      fwd_lay(kFanWeightedEach, D, lanes, npix, 8, c.cl).total <= max_smem_optin() / 2;
    int done = 0;
    while (done < B) {
        const int left = B - done;
        int nb = big, n = left / big * big;   // whole groups of the largest kind first
        if (each && left >= 8) {
            nb = 8;
            n = left / 8 * 8;
        } else if (n == 0) {
            n = left;
            nb = left > 4 ? 8 : left > 2 ? 4 : left;
        }
        const float *sub = c.sub ? c.sub + done * sino : nullptr;
        float *r = (float *)rows, *k = (float *)cols, *o = out + done * sino;
        const float *x = in + done * image;
        int st;
        switch (nb) {
        case 8:
            st = each ? launch_fwd_each(c, x, n, r, k, o, sub) : launch_fwd_passes<KIND, 8>(c, x, n, r, k, o, sub);
            break;
        case 4: st = launch_fwd_passes<KIND, 4>(c, x, n, r, k, o, sub); break;
        case 2: st = launch_fwd_passes<KIND, 2>(c, x, n, r, k, o, sub); break;
        default: st = launch_fwd_passes<KIND, 1>(c, x, n, r, k, o, sub); break;
        }
        if (st != DD_OK) return st;
        c.first = false;
        const int p = plane_slices(nb), planes = (n + nb - 1) / nb * (nb / p);
        rows += planes * plane_bytes(H, W, p);
        cols += planes * plane_bytes(W, H, p);
        done += n;
    }
    return DD_OK;
}

template <int GEOM, int OPK, int NB>
static int launch_adj_as(const dd_geom2d *g, const PlanLayout &P, const char *planb, int B, int V, const float2 *dtab,
                         float *out, const float *base, float scale, int *status, cudaStream_t st) {
    const unsigned ngroups = (unsigned)((B + NB - 1) / NB);
    const dim3 grid((unsigned)((g->width + kTile - 1) / kTile) * ngroups * kAdjCluster, (g->height + kTile - 1) / kTile);
    const AdjSmem S = adj_smem();
    auto kern = k_adj<GEOM, OPK, NB>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S.total) != cudaSuccess)
        return DD_ERR_LAUNCH;
    ProfRec *pr = prof_begin(DD_KERNEL_ADJOINT, st);
    kern<<<grid, kThreads, S.total, st>>>(*g, B, V, (const DdView2 *)(planb + P.views),
                                          (const unsigned char *)(planb + P.amap), (const int2 *)(planb + P.trange),
                                          (const int *)(planb + P.axisv), dtab, out, base, scale, status);
    prof_end(pr, st);
    g_launches++;
    return launch_status();
}

template <int GEOM, int OPK>
static int launch_adj_op(const dd_geom2d *g, const PlanLayout &P, const char *planb, int B, int V, const float2 *dtab,
                         float *out, const float *base, float scale, int *status, cudaStream_t st) {
    if (B == 1) return launch_adj_as<GEOM, OPK, 1>(g, P, planb, B, V, dtab, out, base, scale, status, st);
    return launch_adj_as<GEOM, OPK, kBI>(g, P, planb, B, V, dtab, out, base, scale, status, st);
}

template <int GEOM>
static int launch_adj(int op, const dd_geom2d *g, const PlanLayout &P, const char *planb, int B, int V,
                      const float2 *dtab, float *out, const float *base, float scale, int *status, cudaStream_t st) {
    if (op == DD_OP_PROJ_T) return launch_adj_op<GEOM, 0>(g, P, planb, B, V, dtab, out, base, scale, status, st);
    if (op == DD_OP_BPROJ) return launch_adj_op<GEOM, 1>(g, P, planb, B, V, dtab, out, base, scale, status, st);
    return launch_adj_op<GEOM, 2>(g, P, planb, B, V, dtab, out, base, scale, status, st);
}

// Does one CTA take a line of the parallel beam's adjoint, instead of a cluster
// of kAdjCluster?  It does where the detector tables leave room for no more than
// two CTAs on an SM (the starts of three more are then not hidden by others) and
// the lines fill the chip's waves of them to 0.85.  ms by four / by one, 4 / 8 /
// 12 slices: 300^2, 200 views, 1,200 cells 0.54, 0.95, 1.35 / 0.45, 0.86, 1.26;
// 400^2, 100 views, 1,600 cells 0.41, 0.73, 1.07 / (66 % full) 0.70, 0.72, 0.97.
// With three CTAs and more by one: 256^2, 180 views, 1,024 cells, 12 slices
// 0.75 / 1.18; 512^2, 360 views, 736 cells, 3 slices 0.83 / 1.11.
static bool para_alone(int smem, int npix, long long lines) {
    const int resident = 228 * 1024 / (smem + 1024 + 128);   // of 228 KB an SM, 1 KB goes to each CTA beside its own
    if (resident > 2 || para_pixels(npix) > 4) return false;
    const long long slots = (long long)sm_count() * resident;
    return (double)lines >= 0.85 * (double)((lines + slots - 1) / slots * slots);
}

// Parallel-beam adjoint: the rows' launch writes, the columns' launch adds.
template <int OPK>
static int launch_adj_para(const dd_geom2d *g, const PlanLayout &P, const char *planb, int B, int V, const float2 *dtab,
                           float *out, const float *base, float scale, int *status, cudaStream_t st) {
    const DdLine *lines = (const DdLine *)(planb + P.lines);
    const DdLine *dlines = (const DdLine *)(planb + P.dlines);
    const int *axisv = (const int *)(planb + P.axisv);
    const int W = g->width, H = g->height, D = g->num_det;
    const int nbm = std::min(kBI, B), groups = (B + kBI - 1) / kBI;
    ProfRec *pr = prof_begin(DD_KERNEL_ADJOINT, st);
    for (int axis = 1; axis >= 0; axis--) {
        const int npix = axis ? W : H, nline = axis ? H : W;
        const int smem = para_smem(D, npix, nbm).total;
        if (smem > max_smem_optin()) return DD_ERR_SIZE_OVERFLOW;
        const bool alone = para_alone(smem, npix, (long long)nline * groups);
        const int cl = alone ? 1 : kAdjCluster;
        auto kern = !alone ? k_adj_para<OPK, 0> : para_pixels(npix) <= 2 ? k_adj_para<OPK, 2> : k_adj_para<OPK, 4>;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
            return DD_ERR_LAUNCH;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = (unsigned)cl;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(nline * cl), (unsigned)groups);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = (size_t)smem;
        cfg.stream = st;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        if (cudaLaunchKernelEx(&cfg, kern, *g, B, V, P.nl, axis, axisv, lines, dlines, dtab, out, base, scale, status) !=
            cudaSuccess) {
            (void)cudaGetLastError();
            return DD_ERR_LAUNCH;
        }
    }
    prof_end(pr, st);
    g_launches += 2;
    return launch_status();
}

int launch_det_tables(int geom, int op, const dd_geom2d *g, const char *planb, const float *in, int B,
                      int V, float2 *dtab, int *status, cudaStream_t st) {
    const PlanLayout P = plan_layout(geom == DD_GEOM_PARA ? DD_SCAN_PARA : DD_SCAN_FLAT, g, V);
    const int mode = (op == DD_OP_PROJ_T) ? 0 : 1;
    const float pcx = g->pix_y / g->det_size, pcy = g->pix_x / g->det_size;
    const int nw = B * V;
    ProfRec *pr = prof_begin(DD_KERNEL_TABLES, st);
    k_dettab<<<(nw * 32 + 255) / 256, 256, 0, st>>>(geom, mode, in, B, V, g->num_det,
                                                     (const DdView2 *)(planb + P.views),
                                                     (const float *)(planb + P.dp),
                                                     (const float *)(planb + P.bcoef), pcx, pcy, dtab, status);
    prof_end(pr, st);
    g_launches++;
    return launch_status();
}

int apply_planned(int scan, int op, const dd_geom2d *g, const void *planp, const float *in,
                  float *out, int B, int V, void *ws, size_t wsb, cudaStream_t st,
                  const float *sub = nullptr, const float *base = nullptr, float scale = 1.0f,
                  const dd_tune2d *tune = nullptr) {
    const PlanLayout P = plan_layout(scan, g, V);
    const ApplyLayout A = apply_layout(op, g, B, V);
    if (!ws || wsb < A.total) return DD_ERR_WORKSPACE;
    if (!in || !out || !planp) return DD_ERR_INVALID_ARG;
    const char *planb = (const char *)planp;
    char *wb = (char *)ws;
    int *status = (int *)(wb + A.status);
    const int geom = geom_of(scan);
    if (op_is_forward(op)) {
        FwdCall c;
        c.first = true;
        c.g = g;
        c.geom = geom;
        c.op = op;
        c.V = V;
        c.nl = P.nl;
        int bi;
        fwd_shape(geom, g, tune, &bi, &c.cl);
        c.sh = fwd_lanes(geom, *g);
        c.views = (const DdView2 *)(planb + P.views);
        c.dp = (const float *)(planb + P.dp);
        c.bcoef = (const float *)(planb + P.bcoef);
        c.lines = (const DdLine *)(planb + P.lines);
        c.dlines = geom == DD_GEOM_PARA ? (const DdLine *)(planb + P.dlines) : nullptr;
        c.sub = sub;
        c.status = status;
        c.st = st;
        if (geom == DD_GEOM_PARA) return launch_fwd<kPara>(c, bi == 1, B, in, wb + A.tabx, wb + A.taby, out);
        if (op == DD_OP_BPROJ_TW) return launch_fwd<kFanWeighted>(c, bi == 1, B, in, wb + A.tabx, wb + A.taby, out);
        // (the reason stands at dd2d_prefix.cuh's head; not where the lines'
        // tables are too long for shared memory)
        if (geom == DD_GEOM_ARC && op == DD_OP_PROJ && B <= 2 && prefix_near(*g) &&
            prefix_smem(g->num_det, rs_entries(std::max(g->width, g->height)), B).total <= max_smem_optin()) {
            float2 *tx = (float2 *)(wb + A.tabx), *ty = (float2 *)(wb + A.taby);
            return B == 1 ? launch_prefix<1>(c, B, in, tx, ty, out) : launch_prefix<2>(c, B, in, tx, ty, out);
        }
        if (op != DD_OP_PROJ) return launch_fwd<kFanScaled>(c, bi == 1, B, in, wb + A.tabx, wb + A.taby, out);
        return launch_fwd<kFan>(c, bi == 1, B, in, wb + A.tabx, wb + A.taby, out);
    }
    float2 *dtab = (float2 *)(wb + A.dtab);
    const int ts = launch_det_tables(geom, op, g, planb, in, B, V, dtab, status, st);
    if (ts != DD_OK) return ts;
    if (geom == DD_GEOM_PARA)
        return op == DD_OP_PROJ_T ? launch_adj_para<0>(g, P, planb, B, V, dtab, out, base, scale, status, st)
                                  : launch_adj_para<1>(g, P, planb, B, V, dtab, out, base, scale, status, st);
    if (geom == DD_GEOM_FLAT) return launch_adj<DD_GEOM_FLAT>(op, g, P, planb, B, V, dtab, out, base, scale, status, st);
    return launch_adj<DD_GEOM_ARC>(op, g, P, planb, B, V, dtab, out, base, scale, status, st);
}

}  // namespace dd2

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
using namespace dd2;

extern "C" int dd2d_validate(int scan, int op, const dd_geom2d *g, int batch, int num_view) {
    return validate(scan, op, g, batch, num_view);
}

extern "C" size_t dd2d_plan_bytes(int scan, const dd_geom2d *g, int num_view) {
    if (!g || num_view <= 0) return 0;
    return plan_layout(scan, g, num_view).total;
}

extern "C" size_t dd2d_apply_workspace_bytes(int scan, int op, const dd_geom2d *g, int batch,
                                             int num_view) {
    (void)scan;
    if (!g || batch <= 0 || num_view <= 0) return 0;
    return apply_layout(op, g, batch, num_view).total;
}

extern "C" size_t dd2d_workspace_bytes(int scan, int op, const dd_geom2d *g, int batch, int num_view) {
    if (!g || batch <= 0 || num_view <= 0) return 0;
    return plan_layout(scan, g, num_view, !op_is_forward(op)).total + apply_layout(op, g, batch, num_view).total;
}

extern "C" int dd2d_plan(int scan, const dd_geom2d *g, const float *angles, int num_view, void *planp,
                         size_t plan_bytes, dd_stream_t stream) {
    ddtrace::Range tr("dd2d_plan", scan, -1, false);
    const int st = validate(scan, DD_OP_PROJ, g, 1, num_view);
    if (st != DD_OK) return st;
    return plan(scan, g, angles, num_view, planp, plan_bytes, (cudaStream_t)stream);
}

extern "C" int dd2d_apply(int scan, int op, const dd_geom2d *g, const float *in, float *out,
                          const float *angles, int batch, int num_view, void *workspace,
                          size_t workspace_bytes, dd_stream_t stream) {
    ddtrace::Range tr("dd2d_apply", scan, op, false);
    const int st = validate(scan, op, g, batch, num_view);
    if (st != DD_OK) return st;
    if (!angles || !in || !out) return DD_ERR_INVALID_ARG;
    // a one-shot forward-type call needs no adjoint map in its plan
    const bool with_map = !op_is_forward(op);
    const size_t pb = plan_layout(scan, g, num_view, with_map).total;
    if (!workspace || workspace_bytes < dd2d_workspace_bytes(scan, op, g, batch, num_view))
        return DD_ERR_WORKSPACE;
    const int s1 = plan(scan, g, angles, num_view, workspace, pb, (cudaStream_t)stream, with_map);
    if (s1 != DD_OK) return s1;
    return apply_planned(scan, op, g, workspace, in, out, batch, num_view, (char *)workspace + pb,
                         workspace_bytes - pb, (cudaStream_t)stream);
}

extern "C" int dd2d_apply_planned(int scan, int op, const dd_geom2d *g, const void *planp,
                                  const float *in, float *out, int batch, int num_view,
                                  void *workspace, size_t workspace_bytes, dd_stream_t stream) {
    ddtrace::Range tr("dd2d_apply_planned", scan, op, false);
    const int st = validate(scan, op, g, batch, num_view);
    if (st != DD_OK) return st;
    return apply_planned(scan, op, g, planp, in, out, batch, num_view, workspace, workspace_bytes,
                         (cudaStream_t)stream);
}

extern "C" int dd2d_apply_planned_tuned(int scan, int op, const dd_geom2d *g, const void *planp,
                                        const float *in, float *out, int batch, int num_view,
                                        void *workspace, size_t workspace_bytes, const dd_tune2d *tune,
                                        dd_stream_t stream) {
    ddtrace::Range tr("dd2d_apply_planned", scan, op, false);
    const int st = validate(scan, op, g, batch, num_view);
    if (st != DD_OK) return st;
    return apply_planned(scan, op, g, planp, in, out, batch, num_view, workspace, workspace_bytes,
                         (cudaStream_t)stream, nullptr, nullptr, 1.0f, tune);
}

extern "C" int dd2d_fwd_shape(int scan, const dd_geom2d *g, const dd_tune2d *tune, int *slices, int *cluster) {
    if (!g || !slices || !cluster || scan < DD_SCAN_PARA || scan > DD_SCAN_ARC) return DD_ERR_INVALID_ARG;
    fwd_shape(geom_of(scan), g, tune, slices, cluster);
    return DD_OK;
}

extern "C" size_t dd2d_dc_workspace_bytes(int scan, const dd_geom2d *g, int batch, int num_view) {
    if (!g || batch <= 0 || num_view <= 0) return 0;
    const size_t a = apply_layout(DD_OP_PROJ, g, batch, num_view).total;
    const size_t b = apply_layout(DD_OP_PROJ_T, g, batch, num_view).total;
    (void)scan;
    return a > b ? a : b;
}

extern "C" int dd2d_dc_step(int scan, const dd_geom2d *g, const void *planp, float *x, const float *y,
                            float *resid, float eta, int batch, int num_view, void *workspace,
                            size_t workspace_bytes, dd_stream_t stream) {
    ddtrace::Range tr("dd2d_dc_step", scan, -1, false);
    const int st = validate(scan, DD_OP_PROJ, g, batch, num_view);
    if (st != DD_OK) return st;
    if (!planp || !x || !y || !resid) return DD_ERR_INVALID_ARG;
    if (!workspace || workspace_bytes < dd2d_dc_workspace_bytes(scan, g, batch, num_view)) return DD_ERR_WORKSPACE;
    cudaStream_t s = (cudaStream_t)stream;
    const int s1 = apply_planned(scan, DD_OP_PROJ, g, planp, x, resid, batch, num_view, workspace,
                                 workspace_bytes, s, y);
    if (s1 != DD_OK) return s1;
    return apply_planned(scan, DD_OP_PROJ_T, g, planp, resid, x, batch, num_view, workspace, workspace_bytes,
                         s, nullptr, x, -eta);
}

static int read_word(const void *p, int *status) {
    if (cudaMemcpy(status, p, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return DD_ERR_LAUNCH;
    return DD_OK;
}

extern "C" int dd2d_status(int scan, int op, const dd_geom2d *g, int batch, int num_view, const void *workspace,
                           int *status) {
    if (validate(scan, op, g, batch, num_view) != DD_OK || !workspace || !status) return DD_ERR_INVALID_ARG;
    const size_t pb = plan_layout(scan, g, num_view, !op_is_forward(op)).total;
    return read_word((const char *)workspace + pb + apply_layout(op, g, batch, num_view).status, status);
}

extern "C" int dd2d_planned_status(int op, const dd_geom2d *g, int batch, int num_view, const void *workspace,
                                   int *status) {
    if (!g || batch <= 0 || num_view <= 0 || !workspace || !status) return DD_ERR_INVALID_ARG;
    return read_word((const char *)workspace + apply_layout(op, g, batch, num_view).status, status);
}

// byte offset of the status word of a dd2d_apply call in its workspace (used by
// the no-allocation entry point, whose workspace is the library's own buffer)
size_t dd2d_status_offset(int scan, int op, const dd_geom2d *g, int batch, int num_view) {
    return plan_layout(scan, g, num_view, !op_is_forward(op)).total + apply_layout(op, g, batch, num_view).status;
}

// each translation unit with bounded waits keeps its own sink pointer
int dd2b_set_sink(int *sink);   // dd2d_batch.cu
int dd3_set_sink(int *sink);    // dd3d.cu

extern "C" int dd_set_status_sink(int *sink) {
    int *dev_ptr = nullptr;
    if (sink && cudaHostGetDevicePointer((void **)&dev_ptr, sink, 0) != cudaSuccess) {
        (void)cudaGetLastError();
        return DD_ERR_INVALID_ARG;   // not pinned, device-mapped host memory
    }
    if (dd_set_status_sink_tu(dev_ptr) || dd2b_set_sink(dev_ptr) || dd3_set_sink(dev_ptr)) return DD_ERR_LAUNCH;
    return DD_OK;
}

// named entries (RadonTorch.cpp:1376-1393)
#define DD_NAMED(name, scan, op)                                                              \
    extern "C" int dd_##name(const dd_geom2d *g, const float *in, float *out,                 \
                             const float *angles, int batch, int num_view, void *workspace,   \
                             size_t workspace_bytes, dd_stream_t stream) {                    \
        return dd2d_apply(scan, op, g, in, out, angles, batch, num_view, workspace,           \
                          workspace_bytes, stream);                                           \
    }
DD_NAMED(ProjFanFlatDis2d, DD_SCAN_FLAT, DD_OP_PROJ)
DD_NAMED(ProjTransFanFlatDis2d, DD_SCAN_FLAT, DD_OP_PROJ_T)
DD_NAMED(BackProjFanFlatDis2d, DD_SCAN_FLAT, DD_OP_BPROJ)
DD_NAMED(BackProjTransFanFlatDis2d, DD_SCAN_FLAT, DD_OP_BPROJ_T)
DD_NAMED(BackProjWeightedFanFlatDis2d, DD_SCAN_FLAT, DD_OP_BPROJ_W)
DD_NAMED(BackProjTransWeightedFanFlatDis2d, DD_SCAN_FLAT, DD_OP_BPROJ_TW)
DD_NAMED(ProjFanArcDis2d, DD_SCAN_ARC, DD_OP_PROJ)
DD_NAMED(ProjTransFanArcDis2d, DD_SCAN_ARC, DD_OP_PROJ_T)
DD_NAMED(BackProjFanArcDis2d, DD_SCAN_ARC, DD_OP_BPROJ)
DD_NAMED(BackProjTransFanArcDis2d, DD_SCAN_ARC, DD_OP_BPROJ_T)
DD_NAMED(BackProjWeightedFanArcDis2d, DD_SCAN_ARC, DD_OP_BPROJ_W)
DD_NAMED(BackProjTransWeightedFanArcDis2d, DD_SCAN_ARC, DD_OP_BPROJ_TW)
DD_NAMED(ProjParaDis2d, DD_SCAN_PARA, DD_OP_PROJ)
DD_NAMED(ProjTransParaDis2d, DD_SCAN_PARA, DD_OP_PROJ_T)
DD_NAMED(BackProjParaDis2d, DD_SCAN_PARA, DD_OP_BPROJ)
DD_NAMED(BackProjTransParaDis2d, DD_SCAN_PARA, DD_OP_BPROJ_T)
#undef DD_NAMED

extern "C" const char *dd_status_string(int status) {
    switch (status) {
    case DD_OK: return "ok";
    case DD_ERR_INVALID_ARG: return "invalid argument (null pointer, non-positive size or non-finite geometry)";
    case DD_ERR_SIZE_OVERFLOW: return "sizes exceed the supported index range";
    case DD_ERR_WORKSPACE: return "workspace missing or too small";
    case DD_ERR_LAUNCH: return "CUDA launch or runtime error";
    case DD_ERR_TIMEOUT: return "a bounded device-side wait timed out";
    case DD_ERR_UNSUPPORTED: return "operator not defined for this geometry";
    default: return "unknown status";
    }
}

extern "C" const char *dd_version(void) { return "pridediff_dd 0.4 sm_103a"; }

extern "C" unsigned long long dd_launch_count(void) { return g_launches; }

extern "C" int dd_profile_enable(int on) {
    g_prof = on ? 1 : 0;
    g_prof_used = 0;
    return DD_OK;
}

extern "C" int dd_profile_read(int kind, double *total_ms, int *count) {
    if (!total_ms || !count) return DD_ERR_INVALID_ARG;
    double t = 0.0;
    int n = 0;
    for (int i = 0; i < g_prof_used; i++) {
        if (g_prof_rec[i].kind != kind) continue;
        if (cudaEventSynchronize(g_prof_rec[i].b) != cudaSuccess) return DD_ERR_LAUNCH;
        float ms = 0.0f;
        if (cudaEventElapsedTime(&ms, g_prof_rec[i].a, g_prof_rec[i].b) != cudaSuccess) return DD_ERR_LAUNCH;
        t += ms;
        n++;
    }
    *total_ms = t;
    *count = n;
    return DD_OK;
}
