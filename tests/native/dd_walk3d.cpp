// Host model of the 3-D CUDA kernels' carried walks (test infrastructure): the
// forward's merge of a thread's rows with the slices, a column's pixels summed
// once per slice, and the adjoint's merge of a voxel column's slices with the
// rows of each detector column it meets -- as k_fwd3 and k_adj3 run them, on the
// plan of dd_model3d.cpp and the helpers that the kernels share
// (dd3_pix_bounds, dd3_zb, dd3_rp, dd3_coef, dd3_col_of).
//
// Build: g++ -O2 -std=c++17 -ffp-contract=off -fPIC -shared dd_walk3d.cpp
#include "dd_model3d.cpp"

namespace {

// Overlaps of column k (kk in its walk block) with a line's pixels: the first
// by the linear estimate, settled on the exact boundaries, then in order.
struct Segs {
    int j0 = 0;
    std::vector<float> c;
};
Segs segments(int geom, int family, const dd_geom3d *g, const DdView3 &w, const DdLine &L, const float *dp, int k, int kk,
              float lpos, float parea) {
    Segs s;
    const DdLineHdr h = L.h;
    const float CL = kk == h.idet0 ? h.bound0 : dp[k], CH = dp[k + 1];
    if (h.npiece == 0 || kk < h.idet0 || !(CL < CH)) return s;
    auto bound = [&](int e) {   // boundary e >= i0
        const DdPiece P0 = L.p[0];
        const DdPiece P = L.p[dd_piece_of_index(&L, e, FADD(P0.Q, FMUL((float)(e - P0.gb), P0.dl)))];
        return FADD(P.Q, FMUL((float)(e - P.gb), P.dl));
    };
    const DdPiece P0 = L.p[0];
    const float t = floorf(FMUL(FSUB(CL, P0.Q), P0.invdl)) + (float)(P0.gb + 1);
    int j = (int)fminf(fmaxf(t, (float)h.i0), (float)(h.nend - 1));
    float plo = j > h.i0 ? bound(j - 1) : h.bound0;
    while (j > h.i0 && plo > CL) {
        j--;
        plo = j > h.i0 ? bound(j - 1) : h.bound0;
    }
    float phi = bound(j);
    while (phi <= CL && j < h.nend - 1) {
        plo = phi;
        phi = bound(++j);
    }
    s.j0 = j;
    plo = fmaxf(plo, CL);
    if (!(phi > CL)) return s;
    while (plo < CH) {
        s.c.push_back(dd3_coef(geom, family, g, &w, lpos, j, FSUB(fminf(phi, CH), plo), parea));
        plo = phi;
        if (++j >= h.nend) break;
        phi = bound(j);
    }
    return s;
}

}   // namespace

// rows: detector rows per forward thread (8, 4, 2); slices: per adjoint thread (16, 8)
extern "C" int walk_apply3d(int geom, int op, const dd_geom3d *g, const float *angles, const float *sp, const float *in,
                            float *out, int B, int V, int rows, int slices) {
    const int W = g->width, H = g->height, Dp = g->depth, C = g->num_col, R = g->num_row;
    Plan3 P;
    build_plan(geom, g, angles, sp, V, P);
    const int family = (op == DD_OP_PROJ || op == DD_OP_PROJ_T) ? 0 : (op == DD_OP_BPROJ_W || op == DD_OP_BPROJ_TW) ? 2 : 1;
    const size_t vox = (size_t)W * H * Dp, det = (size_t)V * R * C;
    if (op == DD_OP_PROJ || op == DD_OP_BPROJ_T || op == DD_OP_BPROJ_TW) {
        for (int b = 0; b < B; b++)
            for (int v = 0; v < V; v++) {
                const DdView3 &w = P.views[v];
                const float *dp = &P.dp[(size_t)v * (C + 1)], *rz = &P.rowz[(size_t)v * R * 2];
                for (int k = 0; k < C; k++)
                    for (int r0 = 0; r0 < R; r0 += rows) {
                        const int cc = k / DD3_CHUNK, n = R - r0 < rows ? R - r0 : rows;
                        std::vector<float> a(n), z(n), acc(n, 0.0f);
                        for (int q = 0; q < n; q++)
                            dd3_rp(geom, &w, P.mag[(size_t)v * C + k], rz[2 * (r0 + q)], rz[2 * (r0 + q) + 1], &a[q], &z[q]);
                        for (int l = 0; l < (w.xb ? H : W); l++) {
                            const float *lz = &P.linez[((size_t)v * P.nl + l) * 4];
                            if (!(lz[2] > 0.0f)) continue;
                            const Segs s = segments(geom, family, g, w, P.lines[((size_t)v * P.nl + l) * P.nch + cc], dp, k,
                                                    k - cc * DD3_CHUNK, dd3_line_pos_f(g, &w, l), lz[3]);
                            if (s.c.empty()) continue;
                            // slice i ends at top(i); below the volume and above it nothing is summed
                            auto top = [&](int i) {
                                if (i >= Dp) return (float)INFINITY;
                                const float t = dd3_zb(lz[0], lz[2], i + 1);
                                return i == Dp - 1 ? fminf(t, lz[1]) : t;
                            };
                            auto column = [&](int i) {
                                float x = 0.0f;
                                if (i >= 0 && i < Dp)
                                    for (size_t t = 0; t < s.c.size(); t++)
                                        x = std::fmaf(s.c[t], in[b * vox + vox_index(g, w, i, l, s.j0 + (int)t)], x);
                                return x;
                            };
                            int i = -1;
                            while (i < Dp && !(a[0] < top(i))) i++;
                            float x = column(i), zhi = top(i);
                            for (int q = 0; q < n; q++) {
                                const float w0 = FSUB(fminf(z[q], zhi), a[q]);
                                if (w0 > 0.0f) acc[q] = std::fmaf(w0, x, acc[q]);
                                while (zhi < z[q]) {   // the next slice begins where this one ends
                                    const float lo = zhi;
                                    x = column(++i);
                                    zhi = top(i);
                                    acc[q] = std::fmaf(FSUB(fminf(z[q], zhi), lo), x, acc[q]);
                                }
                            }
                        }
                        for (int q = 0; q < n; q++) {
                            const float scale = family == 0 ? dd3_proj_scale(g, &w, dp[k], dp[k + 1], a[q], z[q]) : w.bp_scale;
                            out[b * det + ((size_t)v * R + r0 + q) * C + (w.flip ? C - 1 - k : k)] = FMUL(acc[q], scale);
                        }
                    }
            }
        return 0;
    }
    for (int b = 0; b < B; b++)
        for (int s0 = 0; s0 < Dp; s0 += slices)
            for (int y = 0; y < H; y++)
                for (int x = 0; x < W; x++) {
                    const int n = Dp - s0 < slices ? Dp - s0 : slices;
                    std::vector<float> acc(n, 0.0f);
                    for (int v = 0; v < V; v++) {
                        const DdView3 &w = P.views[v];
                        const float *dp = &P.dp[(size_t)v * (C + 1)], *rz = &P.rowz[(size_t)v * R * 2];
                        const int line = w.xb ? y : x, j = w.xb ? x : H - 1 - y;
                        const float *lz = &P.linez[((size_t)v * P.nl + line) * 4];
                        if (!(lz[2] > 0.0f)) continue;
                        const float ztop = fminf(dd3_zb(lz[0], lz[2], Dp), lz[1]), zfirst = dd3_zb(lz[0], lz[2], s0);
                        auto row = [&](float mag, int r, float *e0, float *e1) {
                            if (r < R) dd3_rp(geom, &w, mag, rz[2 * r], rz[2 * r + 1], e0, e1);
                            else *e0 = *e1 = INFINITY;
                        };
                        for (int cc = 0; cc < P.nch; cc++) {
                            const DdLine &L = P.lines[((size_t)v * P.nl + line) * P.nch + cc];
                            float PL, PH;
                            if (!dd3_pix_bounds(&L, j, &PL, &PH)) continue;
                            const int c0 = cc * DD3_CHUNK, khi = C - c0 < DD3_CHUNK ? C - c0 : DD3_CHUNK;
                            int k = L.h.idet0;
                            while (k < khi && dp[c0 + k + 1] <= PL) k++;
                            for (; k < khi && (k == L.h.idet0 ? L.h.bound0 : dp[c0 + k]) < PH; k++) {
                                const float CL = k == L.h.idet0 ? L.h.bound0 : dp[c0 + k];
                                const float wd = FSUB(fminf(PH, dp[c0 + k + 1]), fmaxf(PL, CL));
                                const float mag = P.mag[(size_t)v * C + c0 + k];
                                if (!(wd > 0.0f && mag > 0.0f)) continue;
                                const float coef = dd3_coef(geom, family, g, &w, dd3_line_pos_f(g, &w, line), j, wd, lz[3]);
                                auto bin = [&](int r) {
                                    float e0, e1, scale = w.bp_scale;
                                    row(mag, r, &e0, &e1);
                                    if (family == 0) scale = dd3_proj_scale(g, &w, dp[c0 + k], dp[c0 + k + 1], e0, e1);
                                    return FMUL(in[b * det + ((size_t)v * R + r) * C + (w.flip ? C - 1 - c0 - k : c0 + k)], scale);
                                };
                                int r = 0;
                                float e0, e1;
                                row(mag, r, &e0, &e1);
                                while (!(e1 > zfirst) && r < R) row(mag, ++r, &e0, &e1);
                                if (r >= R) continue;
                                float val = bin(r), hi = zfirst;
                                for (int q = 0; q < n; q++) {
                                    const float lo = hi;
                                    hi = fminf(dd3_zb(lz[0], lz[2], s0 + q + 1), ztop);
                                    float t = 0.0f;
                                    const float w0 = FSUB(fminf(e1, hi), fmaxf(e0, lo));
                                    if (w0 > 0.0f) t = std::fmaf(w0, val, t);
                                    while (e1 < hi) {   // the row that ends inside the slice: the next one
                                        row(mag, ++r, &e0, &e1);
                                        if (r < R) val = bin(r);
                                        const float w1 = FSUB(fminf(e1, hi), e0);
                                        if (w1 > 0.0f) t = std::fmaf(w1, val, t);
                                    }
                                    acc[q] = std::fmaf(coef, t, acc[q]);
                                }
                            }
                        }
                    }
                    for (int q = 0; q < n; q++) out[b * vox + ((size_t)(s0 + q) * H + y) * W + x] = acc[q];
                }
    return 0;
}
