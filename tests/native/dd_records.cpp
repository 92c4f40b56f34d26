// Host check of the 2-D walked-line records (test infrastructure): builds a
// line's record with the kernels' own header and evaluates its boundary table
// as the forward's producer warps do (dd2d_fwd.cuh, fill_boundaries), with
// every write checked against the table.
//
// Build: g++ -O2 -std=c++17 -ffp-contract=off -fPIC -shared dd_records.cpp
#include <cmath>
#include <cstring>
#include <vector>

#include "../../pridediff_gb300/csrc/dd_geom2d.cuh"

namespace {
constexpr int kB0 = 4;   // boundary e sits at entry e + kB0

// Writes outside the table (of a line of npix pixels), and the largest
// deviation from the sequential recurrence in ulps of the line's largest value.
int fill(const DdLine &L, int npix, float pint, double *off) {
    const int size = (npix + kB0 + 8 + 3) & ~3;
    std::vector<float> t(size, NAN);
    int bad = 0;
    auto put = [&](int at, float v) {
        if (at < 0 || at >= size) bad++;
        else t[at] = v;
    };
    const int i0 = L.h.i0, nend = L.h.nend, np = L.h.npiece;
    const DdPiece P0 = L.p[0];
    for (int lane = 0; lane < 32; lane++)
        for (int e0 = (i0 & ~7) + 8 * lane; e0 < nend; e0 += 256) {
            const DdPiece P = L.p[dd_piece_of_index(&L, e0, FADD(P0.Q, FMUL((float)(e0 - P0.gb), P0.dl)))];
            for (int i = 0; i < 8; i++) put(e0 + i + kB0, fmaf((float)(e0 - P.gb) + (float)i, P.dl, P.Q));
        }
    for (int lane = 0; lane < np; lane++) {
        const DdPiece P = L.p[lane];
        const int f = lane > 0 ? L.p[lane - 1].gb + 1 : i0, g = f | 7;
        for (int e = f; e <= (P.gb < g ? P.gb : g); e++) put(e + kB0, fmaf((float)(e - P.gb), P.dl, P.Q));
    }
    put(i0 - 1 + kB0, L.h.bound0);
    if (bad) return bad;
    float x = dd_boundary(&L, i0, P0.Q + (float)(i0 - P0.gb) * P0.dl), big = fabsf(x);
    double worst = 0.0;
    std::vector<float> seq;
    for (int e = i0; e < nend; e++) {
        seq.push_back(x);
        big = fmaxf(big, fabsf(x));
        x = x + pint;
    }
    for (int e = i0; e < nend; e++) worst = fmax(worst, fabs((double)t[e + kB0] - (double)seq[e - i0]));
    *off = worst / ldexp(1.0, (int)floor(log2((double)big)) - 23);
    return 0;
}
}   // namespace

// Over all lines of the views: out[0] lines, [1] lines with an ascending pitch,
// [2] records that hold a run outside the line or not in order, [3] writes
// outside the table, [4] lines whose pitch is not positive that keep a record,
// [5] the largest deviation of a table in ulps (rounded up).
extern "C" int records_check(int geom, const dd_geom2d *g, const float *angles, int V, long long *out) {
    std::vector<float> dp(g->num_det + 1), bc(g->num_det);
    for (int i = 0; i < 6; i++) out[i] = 0;
    for (int v = 0; v < V; v++) {
        DdView2 vw;
        dd_view2_setup(geom, g, angles[v], &vw, dp.data(), bc.data());
        const int nline = vw.xb ? g->height : g->width, npix = vw.xb ? g->width : g->height;
        for (int l = 0; l < nline; l++) {
            DdLine L;
            memset(&L, 0, sizeof L);
            DdLineStart st;
            dd_line2_start(geom, g, angles[v], &vw, dp.data(), l, &st);
            dd_line2_setup(geom, g, angles[v], &vw, dp.data(), l, &L, nullptr);
            out[0]++;
            if (st.pint > 0.0f) out[1]++;
            else if (L.h.npiece > 0) out[4]++;
            if (L.h.npiece == 0) continue;
            bool ok = L.h.npiece <= DD_NPMAX && L.p[L.h.npiece - 1].gb == L.h.nend - 1;
            for (int p = 0, from = L.h.i0; p < L.h.npiece; p++) {
                ok = ok && L.p[p].gb >= from && L.p[p].gb < L.h.nend;
                from = L.p[p].gb + 1;
            }
            if (!ok) {
                out[2]++;
                continue;
            }
            double off = 0.0;
            out[3] += fill(L, npix, st.pint, &off);
            if (!(L.h.flags & DD_LINE_SATURATED) && (long long)ceil(off) > out[5]) out[5] = (long long)ceil(off);
        }
    }
    return 0;
}
