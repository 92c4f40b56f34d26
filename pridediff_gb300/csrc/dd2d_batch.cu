// Batched 2-D DD projection over uneven instances, one launch an operator (two
// for the adjoint of a parallel beam) beside the tables'.
//
// An uneven batch is a list of instances, each with its own image size,
// view count, detector count and number of slices (one scan type per batch).
// The reference has no batching beyond folding the batch into gridDim.x with
// one uniform geometry per call (ParaDisCUDA2d.cu:334-337); here every
// instance's geometry plan lives in one plan buffer, the work of all
// instances is cut into items, longest first: forward, one view x a group of
// slices, pulled from a device counter by a persistent grid; adjoint, one
// 32x32 tile (parallel beam: one image line) x a group of slices, a cluster
// each.  The adjoint's item bodies are the single-geometry ones
// (dd2d_kernels.cuh), so its results are identical to per-instance calls; the
// forward's sum the same overlaps (dd2d_fwd.cuh) in another order.  (One or two
// slices of an arc fan are projected by prefix sums in a call of their own,
// dd2d_prefix.cuh: there the two differ by those sums' rounding, 7e-7.)
//
// The data-consistency step x <- x - eta * A^T (A x - y) is four launches:
// image tables, forward items writing the residual A x - y directly, detector
// tables of the residual, adjoint items updating x in place.  No host syncs,
// no allocations: the step is capturable in a CUDA graph.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "dd2d_fwd.cuh"
#include "dd_trace.h"

namespace dd2 {

struct BatchInst {
    dd_geom2d g;
    int V, batch, nl, ps, sh;      // forward items: ps slices (1, 2 or 4), 2^sh lanes a bin
    long long plan_off;            // bytes: instance plan inside the batch plan
    long long img_off, sino_off;   // elements: packed images / sinograms
    long long row_off, col_off;    // bytes: planes of rows / columns in the workspace
    long long dtab_off;            // float2: adjoint tables in the workspace
    long long views, ang, dp, bcoef, lines, dlines, amap, trange, axisv;   // PlanLayout offsets
};

struct BatchLayout {
    size_t desc, fitems, aitems, plans, total;        // plan buffer
    size_t w_tabs, w_dtab, w_resid, w_counter, w_status, w_total;   // workspace
    int nfwd, nadj, nrow, Dmax, nmax;   // items (nrow of the parallel beam's are rows); largest detector and line
    int lanes;   // most lanes that an instance's bins take
    int fi;   // largest instance's slices per forward item
    std::vector<BatchInst> inst;
};

// Most slices per persistent forward item: 4, or fewer where lines of
// thousands of pixels would not leave room for them.
static int fwd_item_limit(int scan, const dd_instance2d *in, int n) {
    int D = 1, npix = 1, lanes = 1;
    for (int i = 0; i < n; i++) {
        D = std::max(D, in[i].geom.num_det);
        lanes = std::max(lanes, in[i].geom.num_det << fwd_lanes(geom_of(scan), in[i].geom));
        npix = std::max(npix, std::max(in[i].geom.width, in[i].geom.height));
    }
    int fi = kBI;
    while (fi > 1 && !fwd_fits(scan == DD_SCAN_PARA ? kPara : kFan, D, lanes, npix, fi, 1, max_smem_optin())) fi /= 2;
    return fi;
}

static BatchLayout batch_layout(int scan, const dd_instance2d *in, int n, int bi) {
    BatchLayout L;
    L.inst.resize(n);
    const int limit = fwd_item_limit(scan, in, n);
    L.fi = 1;
    long long img = 0, sino = 0, tabs = 0, dtab = 0;
    size_t plans = 0;
    L.nfwd = L.nadj = L.nrow = 0;
    L.Dmax = L.lanes = 1;
    L.nmax = 1;
    for (int i = 0; i < n; i++) {
        BatchInst &d = L.inst[i];
        memset(&d, 0, sizeof(d));
        d.g = in[i].geom;
        d.V = in[i].num_view;
        d.batch = in[i].batch;
        const PlanLayout P = plan_layout(scan, &d.g, d.V);
        d.nl = P.nl;
        d.plan_off = (long long)plans;
        plans = align_up(plans + P.total, 256);
        d.views = (long long)P.views;
        d.ang = (long long)P.ang;
        d.dp = (long long)P.dp;
        d.bcoef = (long long)P.bcoef;
        d.lines = (long long)P.lines;
        d.dlines = (long long)P.dlines;
        d.amap = (long long)P.amap;
        d.trange = (long long)P.trange;
        d.axisv = (long long)P.axisv;
        const int W = d.g.width, H = d.g.height, D = d.g.num_det;
        d.img_off = img;
        img += (long long)d.batch * H * W;
        d.sino_off = sino;
        sino += (long long)d.batch * d.V * D;
        d.ps = std::min(limit, d.batch <= 2 ? d.batch : kBI);
        L.fi = std::max(L.fi, d.ps);
        const long long planes = (d.batch + d.ps - 1) / d.ps;
        d.row_off = tabs;
        tabs += planes * (long long)plane_bytes(H, W, d.ps);
        d.col_off = tabs;
        tabs += planes * (long long)plane_bytes(W, H, d.ps);
        d.dtab_off = dtab;
        dtab += ((long long)d.batch * d.V * rs_entries(D) + 1) & ~1LL;
        const int groups = (d.batch + bi - 1) / bi;
        L.nfwd += d.V * ((d.batch + d.ps - 1) / d.ps);
        if (scan == DD_SCAN_PARA) {
            L.nrow += H * groups;
            L.nadj += (H + W) * groups;
        } else {
            L.nadj += ((W + kTile - 1) / kTile) * ((H + kTile - 1) / kTile) * groups;
        }
        L.Dmax = std::max(L.Dmax, D);
        d.sh = fwd_lanes(geom_of(scan), d.g);
        L.lanes = std::max(L.lanes, D << d.sh);
        L.nmax = std::max(L.nmax, std::max(W, H));
    }
    size_t o = 0;
    L.desc = o; o = align_up(o + sizeof(BatchInst) * (size_t)n, 256);
    L.fitems = o; o = align_up(o + sizeof(int4) * (size_t)L.nfwd, 256);
    L.aitems = o; o = align_up(o + sizeof(int4) * (size_t)L.nadj, 256);
    L.plans = o; o = align_up(o + plans, 256);
    L.total = o;
    size_t w = 0;
    L.w_tabs = w; w = align_up(w + (size_t)tabs, 256);
    L.w_dtab = w; w = align_up(w + sizeof(float2) * (size_t)dtab, 256);
    L.w_resid = w; w = align_up(w + sizeof(float) * (size_t)sino, 256);
    L.w_counter = w; w = align_up(w + 2 * sizeof(int), 256);
    L.w_status = w; w = align_up(w + sizeof(int), 256);
    L.w_total = w;
    return L;
}

// ---------------------------------------------------------------------------
// Batched planes of rows and columns (forward) and prefix tables (adjoint);
// one launch each, blockIdx.y = instance
// ---------------------------------------------------------------------------
template <int P>
__device__ __forceinline__ void planes_of(const BatchInst &d, int q, int tile, const float *img, char *tabs, float *t) {
    const int W = d.g.width, H = d.g.height, ntx = (W + 31) / 32;
    plane_tile<P>(img + d.img_off + (size_t)q * P * H * W, min(P, d.batch - q * P), W, H, tile % ntx * 32,
                  tile / ntx * 32, reinterpret_cast<float *>(tabs + d.row_off + q * plane_bytes(H, W, P)),
                  reinterpret_cast<float *>(tabs + d.col_off + q * plane_bytes(W, H, P)),
                  reinterpret_cast<float (*)[33 * P]>(t));
}
__global__ void __launch_bounds__(256)
k_planes_b(const BatchInst *__restrict__ desc, const float *__restrict__ img, char *__restrict__ tabs) {
    __shared__ float t[32 * 33 * 4];
    const BatchInst &d = desc[blockIdx.y];
    const int nt = ((d.g.width + 31) / 32) * ((d.g.height + 31) / 32);
    const int q = blockIdx.x / nt, tile = blockIdx.x - q * nt;
    if (q * d.ps >= d.batch) return;
    if (d.ps == 1) planes_of<1>(d, q, tile, img, tabs, t);
    else if (d.ps == 2) planes_of<2>(d, q, tile, img, tabs, t);
    else planes_of<4>(d, q, tile, img, tabs, t);
}

__global__ void k_dettab_b(int geom, int mode, const BatchInst *__restrict__ desc,
                           const char *__restrict__ plan, size_t plans_off,
                           const float *__restrict__ sino, float2 *__restrict__ dtabs) {
    const BatchInst &d = desc[blockIdx.y];
    const int V = d.V, D = d.g.num_det;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= d.batch * V) return;
    const int b = warp / V, v = warp - b * V;
    const char *pb = plan + plans_off + d.plan_off;
    const DdView2 vw = reinterpret_cast<const DdView2 *>(pb + d.views)[v];
    const float *dpv = reinterpret_cast<const float *>(pb + d.dp) + (size_t)v * (D + 1);
    const float *bc = reinterpret_cast<const float *>(pb + d.bcoef) + (size_t)v * (D + 1);
    const float *s = sino + d.sino_off + ((size_t)b * V + v) * D;
    float2 *t = dtabs + d.dtab_off + (size_t)warp * rs_entries(D);
    const float pc = vw.xb ? d.g.pix_y / d.g.det_size : d.g.pix_x / d.g.det_size;
    warp_prefix_table(D, t, lane, [&](int k, float *g, float *w) {
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

// ---------------------------------------------------------------------------
// Persistent item kernels
// ---------------------------------------------------------------------------
__device__ __forceinline__ int next_item(int *counter) {
    __shared__ int s_item;
    __syncthreads();
    if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
    __syncthreads();
    return s_item;
}

// The forward's clusters: rank 0 takes the next item, the other ranks read its
// index from rank 0's shared memory.  The second barrier keeps rank 0 (and
// its s_item) in place until every rank has read it: past the last item rank
// 0 exits, and a CTA's shared memory must not be read after it has exited.
__device__ __forceinline__ int next_item_cluster(int *counter) {
    __shared__ int s_item;
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    if (cluster.block_rank() == 0 && threadIdx.x == 0) s_item = atomicAdd(counter, 1);
    cluster.sync();
    const int i = *cluster.map_shared_rank(&s_item, 0);
    cluster.sync();
    return i;
}

// CTAs per persistent-forward cluster.  Batches of many short items leave
// little tail to split, and a cluster's start-up costs more than it saves
// (24 uneven one-slice instances: 9.00 ms with clusters of 2, 8.20 ms without,
// of an earlier item body).  The cluster size is a tuning choice
// (dd_tune2d.items_cluster): 1 unless the autotuner finds 2 faster for the
// batch at hand; the result is the same bit for bit.
constexpr int kFwdItemsCluster = 1;

// An item runs with as many slices side by side as its instance has (1, 2 or
// 4): one-slice items in a 4-slice kernel took 6.97 instead of 5.9 ms on 24
// uneven instances of 1 to 3 slices.
static_assert(prods(1) == prods(4) && prods(2) == prods(4), "items of 1, 2 and 4 slices share a CTA's warps");
// WIDE: some instance's bins take more than one lane.
template <int KIND, int NPASS, bool WIDE>
__global__ void __launch_bounds__(fwd_threads(4), NPASS <= 4 ? 3 : 2)
k_fwd_items(const __grid_constant__ FwdLay L, int geom, int op, const BatchInst *__restrict__ desc,
            const int4 *__restrict__ items, int nitems, const char *__restrict__ plan, size_t plans_off,
            const char *__restrict__ tabs, float *__restrict__ out, const float *__restrict__ sub, int cl,
            int *__restrict__ counter, int *__restrict__ status) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ FwdState S;
    fwd_init<KIND, 4>(smem, L, S);
    // the item and its geometry live in shared memory: read where used, they
    // hold no registers across the line loop (the plain forward reads them
    // from kernel parameters)
    __shared__ FwdItem s_it;
    __shared__ dd_geom2d s_g;
    __shared__ int s_ps;
    uint32_t step = 0, nr = 0;
    for (;;) {
        int i;
        if (cl > 1) i = next_item_cluster(counter);
        else i = next_item(counter);
        if (i >= nitems) break;
        if (threadIdx.x == 0) {
            const int4 w = items[i];
            const BatchInst &d = desc[w.x];
            const char *pb = plan + plans_off + d.plan_off;
            const int W = d.g.width, H = d.g.height, q = w.z / d.ps;
            FwdItem it;
            it.v = w.y;
            it.b0 = w.z;
            it.nb = w.w;
            it.V = d.V;
            it.nl = d.nl;
            it.sh = d.sh;
            it.views = reinterpret_cast<const DdView2 *>(pb + d.views);
            it.dp = reinterpret_cast<const float *>(pb + d.dp);
            it.bcoef = reinterpret_cast<const float *>(pb + d.bcoef);
            it.lines = reinterpret_cast<const DdLine *>(pb + d.lines);
            it.dlines = reinterpret_cast<const DdLine *>(pb + d.dlines);
            it.rows = reinterpret_cast<const float *>(tabs + d.row_off + q * plane_bytes(H, W, d.ps));
            it.cols = reinterpret_cast<const float *>(tabs + d.col_off + q * plane_bytes(W, H, d.ps));
            it.rplane = it.cplane = 0;   // one plane per item
            it.out = out + d.sino_off;
            it.sub = sub ? sub + d.sino_off : nullptr;
            s_it = it;
            s_g = d.g;
            s_ps = d.ps;
        }
        __syncthreads();   // every thread passed the barrier above before s_it changes
        const bool ok = s_ps == 1   ? fwd_item<KIND, NPASS, 1, WIDE>(s_g, geom, op, s_it, smem, L, S, step, nr)
                        : s_ps == 2 ? fwd_item<KIND, NPASS, 2, WIDE>(s_g, geom, op, s_it, smem, L, S, step, nr)
                                    : fwd_item<KIND, NPASS, 4, WIDE>(s_g, geom, op, s_it, smem, L, S, step, nr);
        if (!ok) {
            if (threadIdx.x == 0) dd_report_timeout(status);
            break;
        }
    }
}

__device__ __forceinline__ AdjItem adj_item(const BatchInst &d, const int4 w, const char *pb, const float2 *dtabs,
                                            float *out, const float *base, float scale) {
    AdjItem it;
    it.c0 = (w.y & 0xFFFF) * kTile;
    it.r0 = (w.y >> 16) * kTile;
    it.b0 = w.z;
    it.nb = w.w;
    it.V = d.V;
    it.nl = d.nl;
    it.views = reinterpret_cast<const DdView2 *>(pb + d.views);
    it.lines = reinterpret_cast<const DdLine *>(pb + d.lines);
    it.dlines = reinterpret_cast<const DdLine *>(pb + d.dlines);
    it.amap = reinterpret_cast<const unsigned char *>(pb + d.amap);
    it.trange = reinterpret_cast<const int2 *>(pb + d.trange);
    it.axisv = reinterpret_cast<const int *>(pb + d.axisv);
    it.dtab = dtabs + d.dtab_off;
    it.out = out + d.img_off;
    it.base = base ? base + d.img_off : nullptr;
    it.scale = scale;
    return it;
}

// Adjoint items of parallel beams: a cluster per line, the rows by one launch,
// then the columns.
template <int OPK>
__global__ void __cluster_dims__(kAdjCluster, 1, 1) __launch_bounds__(kThreads)
k_adj_items_para(const BatchInst *__restrict__ desc, const int4 *__restrict__ items, int axis,
                 const char *__restrict__ plan, size_t plans_off, const float2 *__restrict__ dtabs,
                 float *__restrict__ out, const float *__restrict__ base, float scale, int Dmax, int nmax,
                 int *__restrict__ status) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ AdjItem s_it;
    __shared__ dd_geom2d s_g;
    if (threadIdx.x == 0) {
        const int4 w = items[blockIdx.x / kAdjCluster];
        const BatchInst &d = desc[w.x];
        s_it = adj_item(d, w, plan + plans_off + d.plan_off, dtabs, out, base, scale);
        s_it.c0 = w.y;
        s_it.r0 = axis;
        s_g = d.g;
    }
    __syncthreads();
    if (!adj_para_line<OPK, 0>(s_g, s_it, smem, para_smem(Dmax, nmax, kBI)) && threadIdx.x == 0) dd_report_timeout(status);
}

// Adjoint items of fan beams: a cluster per item, in the list's order; 4 CTAs
// per SM (64 registers), as the single-geometry adjoint.  Not persistent: the
// clusters behind the resident ones start as these finish, and an item's
// start (its view list, its first copies) then hides behind the SM's other
// CTAs, where a persistent cluster goes through it between two cluster
// barriers (24 uneven instances: 2.60 ms persistent, 2.41 ms so; the map's 14
// GB take 2.06 ms at the copy rate).
template <int GEOM, int OPK>
__global__ void __cluster_dims__(kAdjCluster, 1, 1) __launch_bounds__(kThreads, 4)
k_adj_items(const BatchInst *__restrict__ desc, const int4 *__restrict__ items, const char *__restrict__ plan,
            size_t plans_off, const float2 *__restrict__ dtabs, float *__restrict__ out,
            const float *__restrict__ base, float scale, int *__restrict__ status) {
    extern __shared__ __align__(128) unsigned char smem[];
    const AdjSmem SL = adj_smem();
    __shared__ AdjItem s_it;
    __shared__ dd_geom2d s_g;
    if (threadIdx.x == 0) {
        const int4 w = items[blockIdx.x / kAdjCluster];
        const BatchInst &d = desc[w.x];
        s_it = adj_item(d, w, plan + plans_off + d.plan_off, dtabs, out, base, scale);
        s_g = d.g;
    }
    init_bars(reinterpret_cast<uint64_t *>(smem + SL.bar), kAdjBufs);   // ends with a CTA barrier
    DdPhases ph;
    const bool ok = s_it.nb == 1 ? adj_tile_map<GEOM, OPK, 1>(s_g, s_it, smem, ph)
                                 : adj_tile_map<GEOM, OPK, kBI>(s_g, s_it, smem, ph);
    if (!ok && threadIdx.x == 0) dd_report_timeout(status);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
static int validate_batch(int scan, int op, const dd_instance2d *inst, int n) {
    if (!inst || n <= 0 || n > 65535) return DD_ERR_INVALID_ARG;
    if (op == DD_OP_BPROJ_W || op == DD_OP_BPROJ_TW) return DD_ERR_UNSUPPORTED;
    for (int i = 0; i < n; i++) {
        const int st = validate(scan, op, &inst[i].geom, inst[i].batch, inst[i].num_view);
        if (st != DD_OK) return st;
        if ((inst[i].geom.width + kTile - 1) / kTile > 0xFFFF) return DD_ERR_SIZE_OVERFLOW;
        // the longest lines the persistent forward takes
        const dd_geom2d &g = inst[i].geom;
        if (four_slice_bytes(scan == DD_SCAN_PARA, g.num_det, std::max(g.width, g.height), kFwdItemsCluster) >
            max_smem_optin())
            return DD_ERR_SIZE_OVERFLOW;
    }
    return DD_OK;
}

// Persistent grid: CTAs per SM as the tuning asks, at most as many as fit
// (`fit`, from the kernel's registers and shared memory); 0 = as many as fit.
static int grid_of(const dd_tune2d *t, int nitems, int fit) {
    int per = (t && t->ctas_per_sm > 0) ? t->ctas_per_sm : fit;
    if (per > fit) per = fit;
    if (per < 1) per = 1;
    return std::max(1, std::min(nitems, per * sm_count()));
}

template <typename K>
static int resident_ctas(K kern, int smem, int threads) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, (size_t)smem) != cudaSuccess || n < 1) n = 1;
    return n;
}

template <int KIND, int NPASS, bool WIDE>
static int launch_fwd_items_as(int geom, int op, const BatchLayout &L, const char *planb, char *tabs, float *out,
                               const float *sub, int *counter, int *status, const dd_tune2d *tune, cudaStream_t st) {
    int cl = (tune && tune->items_cluster == 2) ? 2 : kFwdItemsCluster;
    if (cl == 2 && !fwd_fits(KIND, L.Dmax, L.lanes, L.nmax, L.fi, 2, max_smem_optin())) cl = 1;
    const FwdLay S = fwd_lay(KIND, L.Dmax, L.lanes, L.nmax, L.fi, cl);
    auto kern = k_fwd_items<KIND, NPASS, WIDE>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S.total) != cudaSuccess)
        return DD_ERR_LAUNCH;
    // grid_of's CTA count rounded down to whole clusters, at most the clusters
    // that can be resident at once
    const int ctas = grid_of(tune, L.nfwd * cl, resident_ctas(kern, S.total, fwd_threads(4)));
    int clusters = std::max(1, std::min(L.nfwd, ctas / cl));
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)cl;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * cl));
    cfg.blockDim = dim3(fwd_threads(4));
    cfg.dynamicSmemBytes = (size_t)S.total;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (cl > 1) {
        int maxc = 0;
        if (cudaOccupancyMaxActiveClusters(&maxc, (void *)kern, &cfg) == cudaSuccess && maxc > 0)
            clusters = std::min(clusters, maxc);
        else
            (void)cudaGetLastError();
        cfg.gridDim = dim3((unsigned)(clusters * cl));
    }
    ProfRec *pr = prof_begin(DD_KERNEL_FORWARD, st);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, S, geom, op, (const BatchInst *)(planb + L.desc),
                                             (const int4 *)(planb + L.fitems), L.nfwd, planb, L.plans, (const char *)tabs,
                                             out, sub, cl, counter, status);
    prof_end(pr, st);
    count_launches(1);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return DD_ERR_LAUNCH;
    }
    return launch_status();
}

template <int KIND>
static int launch_fwd_items(int geom, int op, const BatchLayout &L, const char *planb, const float *in, char *tabs,
                            float *out, const float *sub, int *counter, int *status, const dd_tune2d *tune,
                            cudaStream_t st) {
    int maxt = 1;
    for (const BatchInst &d : L.inst)
        maxt = std::max(maxt, ((d.batch + d.ps - 1) / d.ps) * ((d.g.width + 31) / 32) * ((d.g.height + 31) / 32));
    ProfRec *pr = prof_begin(DD_KERNEL_TABLES, st);
    k_planes_b<<<dim3((unsigned)maxt, (unsigned)L.inst.size()), 256, 0, st>>>((const BatchInst *)(planb + L.desc), in, tabs);
    prof_end(pr, st);
    count_launches(1);
    if (cudaMemsetAsync(counter, 0, 2 * sizeof(int), st) != cudaSuccess) return DD_ERR_LAUNCH;
    bool wide = false;
    for (const BatchInst &d : L.inst) wide = wide || d.sh > 0;
    const int passes = pass_class(L.lanes);
    if (wide) {   // (few classes: batches with coarse detectors)
        if (passes <= 2) return launch_fwd_items_as<KIND, 2, true>(geom, op, L, planb, tabs, out, sub, counter, status, tune, st);
        if (passes <= 4) return launch_fwd_items_as<KIND, 4, true>(geom, op, L, planb, tabs, out, sub, counter, status, tune, st);
        return launch_fwd_items_as<KIND, 8, true>(geom, op, L, planb, tabs, out, sub, counter, status, tune, st);
    }
    switch (passes) {
    case 1: return launch_fwd_items_as<KIND, 1, false>(geom, op, L, planb, tabs, out, sub, counter, status, tune, st);
    case 2: return launch_fwd_items_as<KIND, 2, false>(geom, op, L, planb, tabs, out, sub, counter, status, tune, st);
    case 3: return launch_fwd_items_as<KIND, 3, false>(geom, op, L, planb, tabs, out, sub, counter, status, tune, st);
    case 4: return launch_fwd_items_as<KIND, 4, false>(geom, op, L, planb, tabs, out, sub, counter, status, tune, st);
    default: return launch_fwd_items_as<KIND, 8, false>(geom, op, L, planb, tabs, out, sub, counter, status, tune, st);
    }
}

template <int GEOM>
static int launch_adj_items(int op, const BatchLayout &L, const char *planb, const float2 *dtabs,
                            float *out, const float *base, float scale, int *status, cudaStream_t st) {
    const BatchInst *desc = (const BatchInst *)(planb + L.desc);
    const int4 *items = (const int4 *)(planb + L.aitems);
    ProfRec *pr = prof_begin(DD_KERNEL_ADJOINT, st);
    if constexpr (GEOM == DD_GEOM_PARA) {
        auto kern = (op == DD_OP_PROJ_T) ? k_adj_items_para<0> : k_adj_items_para<1>;
        const int smem = para_smem(L.Dmax, L.nmax, kBI).total;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
            return DD_ERR_LAUNCH;
        for (int axis = 1; axis >= 0; axis--) {
            const int4 *from = axis ? items : items + L.nrow;
            const int n = axis ? L.nrow : L.nadj - L.nrow;
            kern<<<(unsigned)n * kAdjCluster, kThreads, smem, st>>>(desc, from, axis, planb, L.plans, dtabs, out, base, scale,
                                                                   L.Dmax, L.nmax, status);
        }
        count_launches(1);
    } else {
        const AdjSmem S = adj_smem();
        auto kern = (op == DD_OP_PROJ_T) ? k_adj_items<GEOM, 0> : k_adj_items<GEOM, 1>;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S.total) != cudaSuccess)
            return DD_ERR_LAUNCH;
        kern<<<(unsigned)L.nadj * kAdjCluster, kThreads, S.total, st>>>(desc, items, planb, L.plans, dtabs, out, base,
                                                                       scale, status);
    }
    prof_end(pr, st);
    count_launches(1);
    return launch_status();
}

// forward of all instances: out = A in (- sub)
static int batch_forward(int scan, int op, const BatchLayout &L, const char *planb, const float *in,
                         float *out, const float *sub, char *wb, const dd_tune2d *tune, cudaStream_t st) {
    const int geom = geom_of(scan);
    char *tabs = wb + L.w_tabs;
    int *counter = (int *)(wb + L.w_counter);
    int *status = (int *)(wb + L.w_status);
    if (geom == DD_GEOM_PARA) return launch_fwd_items<kPara>(geom, op, L, planb, in, tabs, out, sub, counter, status, tune, st);
    if (op != DD_OP_PROJ) return launch_fwd_items<kFanScaled>(geom, op, L, planb, in, tabs, out, sub, counter, status, tune, st);
    return launch_fwd_items<kFan>(geom, op, L, planb, in, tabs, out, sub, counter, status, tune, st);
}

// adjoint of all instances: out = base + scale * (A^T in)   (base may be null)
static int batch_adjoint(int scan, int op, const BatchLayout &L, const char *planb, const float *in,
                         float *out, const float *base, float scale, char *wb, cudaStream_t st) {
    const int geom = geom_of(scan);
    float2 *dtabs = (float2 *)(wb + L.w_dtab);
    int *status = (int *)(wb + L.w_status);
    const BatchInst *desc = (const BatchInst *)(planb + L.desc);
    int maxw = 1;
    for (const BatchInst &d : L.inst) maxw = std::max(maxw, d.batch * d.V);
    const int n = (int)L.inst.size();
    ProfRec *pr = prof_begin(DD_KERNEL_TABLES, st);
    k_dettab_b<<<dim3((maxw * 32 + 255) / 256, n), 256, 0, st>>>(geom, op == DD_OP_PROJ_T ? 0 : 1, desc,
                                                                  planb, L.plans, in, dtabs);
    prof_end(pr, st);
    count_launches(1);
    if (geom == DD_GEOM_PARA) return launch_adj_items<DD_GEOM_PARA>(op, L, planb, dtabs, out, base, scale, status, st);
    if (geom == DD_GEOM_FLAT) return launch_adj_items<DD_GEOM_FLAT>(op, L, planb, dtabs, out, base, scale, status, st);
    return launch_adj_items<DD_GEOM_ARC>(op, L, planb, dtabs, out, base, scale, status, st);
}

}  // namespace dd2

using namespace dd2;

extern "C" size_t dd2d_batch_plan_bytes(int scan, const dd_instance2d *inst, int n) {
    if (validate_batch(scan, DD_OP_PROJ, inst, n) != DD_OK) return 0;
    return batch_layout(scan, inst, n, kBI).total;
}

extern "C" size_t dd2d_batch_workspace_bytes(int scan, const dd_instance2d *inst, int n) {
    if (validate_batch(scan, DD_OP_PROJ, inst, n) != DD_OK) return 0;
    return batch_layout(scan, inst, n, kBI).w_total;
}

extern "C" int dd2d_batch_plan(int scan, const dd_instance2d *inst, int n, const float *const *angles,
                               void *planp, size_t plan_bytes, const dd_tune2d *tune, dd_stream_t stream) {
    ddtrace::Range tr("dd2d_batch_plan", scan, -1, false);
    const int vs = validate_batch(scan, DD_OP_PROJ, inst, n);
    if (vs != DD_OK) return vs;
    if (!angles || !planp) return DD_ERR_INVALID_ARG;
    for (int i = 0; i < n; i++)
        if (!angles[i]) return DD_ERR_INVALID_ARG;
    BatchLayout L = batch_layout(scan, inst, n, kBI);
    if (plan_bytes < L.total) return DD_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    char *pb = (char *)planp;
    // work items; longest first unless the tuning asks for instance order
    struct Item {
        int4 w;
        long long cost;
    };
    std::vector<Item> fw, aw, ac;   // ac: the parallel beam's columns
    fw.reserve(L.nfwd);
    aw.reserve(L.nadj);
    for (int i = 0; i < n; i++) {
        const BatchInst &d = L.inst[i];
        const int W = d.g.width, H = d.g.height, D = d.g.num_det;
        for (int b0 = 0; b0 < d.batch; b0 += d.ps) {
            const int nb = std::min(d.ps, d.batch - b0);
            for (int v = 0; v < d.V; v++)
                fw.push_back({make_int4(i, v, b0, nb), (long long)std::max(W, H) * (D + 1) * nb});
        }
        for (int b0 = 0; b0 < d.batch; b0 += kBI) {
            const int nb = std::min(kBI, d.batch - b0);
            if (scan == DD_SCAN_PARA) {
                for (int y = 0; y < H; y++) aw.push_back({make_int4(i, y, b0, nb), (long long)d.V * W * nb});
                for (int x = 0; x < W; x++) ac.push_back({make_int4(i, x, b0, nb), (long long)d.V * H * nb});
                continue;
            }
            for (int ty = 0; ty < (H + kTile - 1) / kTile; ty++)
                for (int tx = 0; tx < (W + kTile - 1) / kTile; tx++)
                    aw.push_back({make_int4(i, tx | (ty << 16), b0, nb), (long long)d.V * nb});
        }
    }
    const bool lpt = !tune || tune->lpt_order != 0;
    if (lpt) {
        std::stable_sort(fw.begin(), fw.end(), [](const Item &a, const Item &b) { return a.cost > b.cost; });
        std::stable_sort(aw.begin(), aw.end(), [](const Item &a, const Item &b) { return a.cost > b.cost; });
        std::stable_sort(ac.begin(), ac.end(), [](const Item &a, const Item &b) { return a.cost > b.cost; });
    }
    aw.insert(aw.end(), ac.begin(), ac.end());
    std::vector<int4> fi(fw.size()), ai(aw.size());
    for (size_t k = 0; k < fw.size(); k++) fi[k] = fw[k].w;
    for (size_t k = 0; k < aw.size(); k++) ai[k] = aw[k].w;
    // descriptors and item lists (plan time only: synchronous copies)
    if (cudaMemcpyAsync(pb + L.desc, L.inst.data(), sizeof(BatchInst) * n, cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(pb + L.fitems, fi.data(), sizeof(int4) * fi.size(), cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(pb + L.aitems, ai.data(), sizeof(int4) * ai.size(), cudaMemcpyHostToDevice, st) != cudaSuccess)
        return DD_ERR_LAUNCH;
    for (int i = 0; i < n; i++) {
        const BatchInst &d = L.inst[i];
        const int s2 = plan(scan, &d.g, angles[i], d.V, pb + L.plans + d.plan_off,
                            plan_layout(scan, &d.g, d.V).total, st);
        if (s2 != DD_OK) return s2;
    }
    if (cudaStreamSynchronize(st) != cudaSuccess) return DD_ERR_LAUNCH;
    return DD_OK;
}

extern "C" int dd2d_batch_apply(int scan, int op, const dd_instance2d *inst, int n, const void *planp,
                                const float *in, float *out, void *ws, size_t wsb, const dd_tune2d *tune,
                                dd_stream_t stream) {
    ddtrace::Range tr("dd2d_batch_apply", scan, op, false);
    const int vs = validate_batch(scan, op, inst, n);
    if (vs != DD_OK) return vs;
    if (!planp || !in || !out) return DD_ERR_INVALID_ARG;
    const BatchLayout L = batch_layout(scan, inst, n, kBI);
    if (!ws || wsb < L.w_total) return DD_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    char *wb = (char *)ws;
    if (cudaMemsetAsync(wb + L.w_status, 0, sizeof(int), st) != cudaSuccess) return DD_ERR_LAUNCH;
    if (op_is_forward(op))
        return batch_forward(scan, op, L, (const char *)planp, in, out, nullptr, wb, tune, st);
    return batch_adjoint(scan, op, L, (const char *)planp, in, out, nullptr, 1.0f, wb, st);
}

extern "C" int dd2d_batch_dc_step(int scan, const dd_instance2d *inst, int n, const void *planp, float *x,
                                  const float *y, float eta, void *ws, size_t wsb, const dd_tune2d *tune,
                                  dd_stream_t stream) {
    ddtrace::Range tr("dd2d_batch_dc_step", scan, -1, false);
    const int vs = validate_batch(scan, DD_OP_PROJ, inst, n);
    if (vs != DD_OK) return vs;
    if (!planp || !x || !y) return DD_ERR_INVALID_ARG;
    const BatchLayout L = batch_layout(scan, inst, n, kBI);
    if (!ws || wsb < L.w_total) return DD_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    char *wb = (char *)ws;
    float *resid = (float *)(wb + L.w_resid);
    const char *pb = (const char *)planp;
    if (cudaMemsetAsync(wb + L.w_status, 0, sizeof(int), st) != cudaSuccess) return DD_ERR_LAUNCH;
    int s1 = batch_forward(scan, DD_OP_PROJ, L, pb, x, resid, y, wb, tune, st);
    if (s1 != DD_OK) return s1;
    return batch_adjoint(scan, DD_OP_PROJ_T, L, pb, resid, x, x, -eta, wb, st);
}

int dd2b_set_sink(int *sink) { return dd_set_status_sink_tu(sink); }

extern "C" int dd2d_batch_status(int scan, const dd_instance2d *inst, int n, const void *ws, int *status) {
    if (validate_batch(scan, DD_OP_PROJ, inst, n) != DD_OK || !ws || !status) return DD_ERR_INVALID_ARG;
    const BatchLayout L = batch_layout(scan, inst, n, kBI);
    if (cudaMemcpy(status, (const char *)ws + L.w_status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
        return DD_ERR_LAUNCH;
    return DD_OK;
}
