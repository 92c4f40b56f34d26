// FBP detector-row filtering with the cosine weight fused.
//
// deeprecon's filtered_backprojection (projector.py:192-213 for 2-D fan and
// parallel beams, :368-390 for cone beams, :554-563 for spirals) weights the
// sinogram and filters every detector row with a 2D - 1 tap kernel:
//
//     nn.functional.conv2d(sino * weight, filter, padding=(0, D - 1))
//
// (conv3d for the 3-D geometries), i.e. the cross-correlation
//
//     out[i][k] = sum_n taps[n - k + D - 1] * (weight[i % wrows][n] * in[i][n])
//
// over the D bins n of row i, before the weighted DD back-projection.  One
// kernel does both: a CTA stages the taps and the weighted bins of kRows rows
// in shared memory and each thread accumulates kOut adjacent outputs of every
// row.  The products are rounded once as the reference's `sino * weight` is;
// the sums run in FP32 in bin order.
//
// Bound by the FP32 pipe: 2 D^2 flops a row.  Rows go in pairs through packed
// multiply-adds, the rows of a bin lie side by side (one broadcast load), and
// four bins at a time share one load of four taps, which slide through a
// register window: 32 packed multiply-adds, 5 loads and the taps' copies, where
// a scalar multiply-add each, a load per row and bin and a 4-way bank conflict
// per tap cost 84 instructions and 32 wavefronts.  11,520 rows of 736 bins:
// 0.353 -> 0.251 ms (35 -> 50 TFLOP/s); 2,880 rows of 768: about 40 us less.
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/pridediff_dd.h"
#include "dd_trace.h"

namespace dd2 {
struct ProfRec;
ProfRec *prof_begin(int kind, cudaStream_t st);
void prof_end(ProfRec *r, cudaStream_t st);
void count_launches(int n);
}   // namespace dd2

namespace ddfbp {

constexpr int kThreads = 256;   // at most
constexpr int kRows = 4;   // rows per CTA (the taps are staged once for them)
constexpr int kOut = 4;    // adjacent outputs per thread and row, and bins per step

// Taps start at an offset that puts the one a step begins with, D - 1 + n - k
// for n and k multiples of 4, on 16 bytes, with room for 3 below them.
__host__ __device__ inline int taps_offset(int D) { return 4 + (-(D - 1) & 3); }
__host__ __device__ inline int taps_stride(int D) { return (taps_offset(D) + 2 * D - 1 + 3) & ~3; }

inline size_t smem_bytes(int D) { return sizeof(float) * ((size_t)taps_stride(D) + (size_t)kRows * D); }

__device__ __forceinline__ unsigned long long both(float t) {
    const unsigned long long u = __float_as_uint(t);
    return u | (u << 32);
}
__device__ __forceinline__ void fma2(unsigned long long &a, unsigned long long t, unsigned long long x) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a) : "l"(t), "l"(x));
}

// weight == nullptr: unit weight.
__global__ void __launch_bounds__(kThreads)
k_fbp_filter(const float *__restrict__ in, float *__restrict__ out, const float *__restrict__ weight, int wrows,
             const float *__restrict__ taps, long long rows, int D) {
    extern __shared__ __align__(16) float sm[];
    const int off = taps_offset(D);
    float *st = sm;                                                     // taps, 2D - 1 from off
    ulonglong2 *sx = reinterpret_cast<ulonglong2 *>(sm + taps_stride(D));   // [bin]: kRows weighted rows, in pairs
    const int tid = threadIdx.x, nt = blockDim.x;
    const long long row0 = (long long)blockIdx.x * kRows;
    const int nr = (int)min((long long)kRows, rows - row0);
    if (tid < off) st[tid] = 0.0f;
    for (int i = tid; i < 2 * D - 1; i += nt) st[off + i] = taps[i];
    const float *src[kRows], *wr[kRows];
#pragma unroll
    for (int r = 0; r < kRows; r++) {
        src[r] = in + (row0 + min(r, nr - 1)) * D;
        wr[r] = weight ? weight + ((row0 + min(r, nr - 1)) % wrows) * D : nullptr;
    }
    for (int n = tid; n < D; n += nt) {
        float v[kRows];
#pragma unroll
        for (int r = 0; r < kRows; r++) v[r] = r < nr ? (weight ? __fmul_rn(src[r][n], wr[r][n]) : src[r][n]) : 0.0f;
        reinterpret_cast<float4 *>(sx)[n] = make_float4(v[0], v[1], v[2], v[3]);
    }
    __syncthreads();
    for (int k0 = tid * kOut; k0 < D; k0 += nt * kOut) {
        // output k0 + i takes bin n by tap D - 1 + n - k0 - i, i.e. by
        // win[3 + j - i] for bin n + j of a step that starts at tap tp[0].
        // (Outputs past the row's end read the zeros below the taps; they are
        // not written.)
        const float *tp = st + off + D - 1 - k0;
        unsigned long long acc[kOut][2], win[7];
#pragma unroll
        for (int i = 0; i < kOut; i++) acc[i][0] = acc[i][1] = 0ull;
#pragma unroll
        for (int i = 0; i < 3; i++) win[i] = both(tp[i - 3]);
        const int steps = D / 4;
#pragma unroll 2
        for (int s = 0; s < steps; s++) {
            const float4 t = *reinterpret_cast<const float4 *>(tp + 4 * s);
            win[3] = both(t.x);
            win[4] = both(t.y);
            win[5] = both(t.z);
            win[6] = both(t.w);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const ulonglong2 x = sx[4 * s + j];
#pragma unroll
                for (int i = 0; i < kOut; i++) {
                    fma2(acc[i][0], win[3 + j - i], x.x);
                    fma2(acc[i][1], win[3 + j - i], x.y);
                }
            }
#pragma unroll
            for (int i = 0; i < 3; i++) win[i] = win[i + 4];
        }
        for (int n = 4 * steps; n < D; n++) {   // the last bins, one at a time
            const ulonglong2 x = sx[n];
#pragma unroll
            for (int i = 0; i < kOut; i++) {
                const unsigned long long t = both(tp[n - i]);
                fma2(acc[i][0], t, x.x);
                fma2(acc[i][1], t, x.y);
            }
        }
#pragma unroll
        for (int r = 0; r < kRows; r++) {
            if (r >= nr) break;
#pragma unroll
            for (int i = 0; i < kOut; i++)
                if (k0 + i < D)
                    out[(row0 + r) * D + k0 + i] = __uint_as_float((unsigned)(acc[i][r >> 1] >> (r & 1 ? 32 : 0)));
        }
    }
}

}   // namespace ddfbp

using namespace ddfbp;

extern "C" int dd_fbp_filter(const float *in, float *out, const float *weight, int wrows, const float *taps,
                             long long rows, int num_det, dd_stream_t stream) {
    ddtrace::Range tr("dd_fbp_filter");
    if (!in || !out || !taps || rows <= 0 || num_det <= 0 || (weight && wrows <= 0)) return DD_ERR_INVALID_ARG;
    if (num_det > 8192 || (rows + kRows - 1) / kRows > 2147483647LL) return DD_ERR_SIZE_OVERFLOW;
    const size_t sb = smem_bytes(num_det);
    if (cudaFuncSetAttribute(k_fbp_filter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sb) != cudaSuccess)
        return DD_ERR_LAUNCH;
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned grid = (unsigned)((rows + kRows - 1) / kRows);
    dd2::ProfRec *pr = dd2::prof_begin(DD_KERNEL_FILTER, st);
    const int threads = std::min(kThreads, ((num_det + kOut - 1) / kOut + 31) / 32 * 32);
    k_fbp_filter<<<grid, threads, sb, st>>>(in, out, weight, weight ? wrows : 1, taps, rows, num_det);
    dd2::prof_end(pr, st);
    dd2::count_launches(1);
    return cudaGetLastError() == cudaSuccess ? DD_OK : DD_ERR_LAUNCH;
}
