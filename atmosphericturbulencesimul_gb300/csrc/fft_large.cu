// fft_large.cu -- unnormalised 2-D DFT of 4096^2 and 8192^2 complex grids,
// the transform behind master screens of that size (the reference's
// make_master_turbulence_screen, AtmosphericTurbulence.c:643-855, calls
// do2dfft on the full M x M spectrum, :783).
//
// Rows: one CTA of 256 threads owns one row; each thread holds M / 256 values
// in registers and the engine's Stockham stages (fft3_ct) run three in-register
// radix stages (16 x 16 x 16 for 4096, 32 x 16 x 16 for 8192) with two
// exchanges through one padded shared row (68 KB at 8192).
// Columns: in place of the array's layout, as two passes of short transforms
// (M = N1 N2, k_fft_cols_1 / k_fft_cols_2), so nothing is transposed.
// Three passes, each one read and one write of the grid: 3 x 2 x 8 M^2 bytes,
// 3.2 GB at 8192^2.
// The whole-row plans run a little faster with scalar butterflies (rows of 8192^2
// 194 us, 197 with packed ones).
#define AW_SCALAR_BUTTERFLY 1
#include "aux_kernels.cuh"
#include "pass_impl.cuh"

namespace atmwfs {

// One row per CTA; ds = -1 forward, +1 inverse.  HBM should bound it (1.07 GB at
// 8192^2, 158 us); it takes 194 us (4096^2: 49).  The last radix stage leaves
// neighbouring outputs in neighbouring threads, so they are stored from
// registers: a third exchange to reorder them cost 25 us.  With the stages
// compiled for the size and the registers bounded for kRowCtas CTAs per SM the
// exchange addresses are constants and a second row's loads run under the
// first's stages: 305 us on the runtime stage loop, 267 unbounded (one CTA of
// 183 registers); three CTAs per SM spill at 8192 (362).
template <int N> constexpr int kRowCtas = N > 4096 ? 2 : 4;
template <int N>
__global__ void __launch_bounds__(Plan<N>::T, kRowCtas<N>) k_fft_row_plan(const float2* __restrict__ in,
                                                                          float2* __restrict__ out,
                                                                          const float2* __restrict__ tw, float ds)
{
    constexpr int T = Plan<N>::T, E = Plan<N>::E, RL = last_radix<N>();
    extern __shared__ float4 big_smem[];
    float2* xrow = reinterpret_cast<float2*>(big_smem);
    const int t = threadIdx.x;
    const size_t row = (size_t)blockIdx.x * N;
    float2 v[E];
#pragma unroll
    for (int e = 0; e < E; e++) v[e] = in[row + t + e * T];
    if (ds > 0.0f) conj_all<E>(v);  // inverse = conj(forward(conj))
    fft3_ct<N, T, E, Stages<N>::R0, Stages<N>::R1, Stages<N>::R2>(v, xrow, t, tw + tw_offset<N>(0, 1), tw + tw_offset<N>(0, 2));
    if (ds > 0.0f) conj_all<E>(v);
#pragma unroll
    for (int s = 0; s < E; s++) out[row + last_index<N, T, RL>(t, s)] = v[s];
}

// Column transforms of the M x M grid, M = N1 N2:
//   X[k1 + N1 k2] = sum_y2 W_N2^(y2 k2) W_M^(y2 k1) sum_y1 W_N1^(y1 k1) x[N2 y1 + y2].
// HBM bounds both passes (1.07 GB each at 8192^2), which is why they replace
// the 32 x 32-tile transposes around a second row pass: those streamed the
// grid twice more without computing anything (2 x 154 us of 881).  A CTA takes
// kCols neighbouring columns of one short transform with the columns along the
// lanes, so that every access is a 128-byte run of a row.  (With a column's
// threads side by side in a warp the accesses are 32-byte pieces, and the rate
// of L2 requests bounds the passes: 526 and 396 us.)
constexpr int kCols = 16;

// One transform of length N (two-stage plan) per column c of the CTA: thread t
// of the column holds x[t + T e] and ends with X[last_index(t, s)].  Stage
// buffer [N][kCols]: a half-warp's 16 columns are one 128-byte row of it.
template <int N>
__device__ __forceinline__ void fft_col(float2 (&v)[Plan<N>::E], float2* buf, int t, int c, const float2* __restrict__ tw)
{
    constexpr int T = Plan<N>::T, E = Plan<N>::E, RA = Stages<N>::R0, RB = Stages<N>::R1;
    static_assert(Stages<N>::S == 2 && E == RA, "one first-stage work item per thread");
    stage_dft<E, RA, -1>(v);
#pragma unroll
    for (int q = 0; q < RA; q++) buf[(t * RA + q) * kCols + c] = v[q];
    __syncthreads();
#pragma unroll
    for (int w = 0; w < E / RB; w++)
#pragma unroll
        for (int r = 0; r < RB; r++) v[w * RB + r] = buf[(t + T * w + r * (N / RB)) * kCols + c];
    stage_twiddle_rt<N, T, E, RB>(v, t, tw + tw_offset<N>(0, 1), RA);
    stage_dft<E, RB, -1>(v);
}

// Pass 1: the inner sum for one y2 (blockIdx.y), times W_M^(y2 k1), in place.
template <int N1, int N2>
__global__ void __launch_bounds__(Plan<N1>::T * kCols) k_fft_cols_1(float2* __restrict__ a, const float2* __restrict__ tw,
                                                                    const float2* __restrict__ wm, float ds)
{
    constexpr int M = N1 * N2, T = Plan<N1>::T, E = Plan<N1>::E, RL = last_radix<N1>();
    __shared__ float2 buf[N1 * kCols];
    const int t = threadIdx.x / kCols, c = threadIdx.x % kCols, y2 = blockIdx.y;
    float2* col = a + (size_t)y2 * M + blockIdx.x * kCols + c;
    float2 v[E];
#pragma unroll
    for (int e = 0; e < E; e++) v[e] = col[(size_t)(t + e * T) * N2 * M];
    if (ds > 0.0f) conj_all<E>(v);
    fft_col<N1>(v, buf, t, c, tw);
#pragma unroll
    for (int s = 0; s < E; s++) {
        const int k1 = last_index<N1, T, RL>(t, s);
        float2 r = cmul(v[s], __ldg(wm + y2 * k1));  // y2 k1 < M
        if (ds > 0.0f) r.y = -r.y;
        col[(size_t)k1 * N2 * M] = r;
    }
}

// Pass 2: the outer sum for one k1 (blockIdx.y); output row k1 + N1 k2.
template <int N1, int N2>
__global__ void __launch_bounds__(Plan<N2>::T * kCols) k_fft_cols_2(const float2* __restrict__ a, float2* __restrict__ out,
                                                                    const float2* __restrict__ tw, float ds)
{
    constexpr int M = N1 * N2, T = Plan<N2>::T, E = Plan<N2>::E, RL = last_radix<N2>();
    __shared__ float2 buf[N2 * kCols];
    const int t = threadIdx.x / kCols, c = threadIdx.x % kCols, k1 = blockIdx.y;
    const size_t x = (size_t)blockIdx.x * kCols + c;
    float2 v[E];
#pragma unroll
    for (int e = 0; e < E; e++) v[e] = a[((size_t)k1 * N2 + t + e * T) * M + x];
    if (ds > 0.0f) conj_all<E>(v);
    fft_col<N2>(v, buf, t, c, tw);
    if (ds > 0.0f) conj_all<E>(v);
#pragma unroll
    for (int s = 0; s < E; s++) out[((size_t)k1 + (size_t)N1 * last_index<N2, T, RL>(t, s)) * M + x] = v[s];
}

bool fft2d_large_supported(long M) { return M == 4096 || M == 8192; }

template <int N1, int N2>
static cudaError_t fft2d_large_t(const float2* in, float2* out, float2* tmp, int sign, cudaStream_t st)
{
    constexpr int M = N1 * N2;
    const float2 *tw = stage_twiddles(M), *tw1 = stage_twiddles(N1), *tw2 = stage_twiddles(N2), *wm = circle_table(M);
    if (!tw || !tw1 || !tw2 || !wm) return cudaErrorMemoryAllocation;
    const int smem = row_stride<M>() * (int)sizeof(float2);
    cudaError_t e = cudaFuncSetAttribute(k_fft_row_plan<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const float ds = sign < 0 ? -1.0f : 1.0f;
    k_fft_row_plan<M><<<M, Plan<M>::T, smem, st>>>(in, tmp, tw, ds);
    k_fft_cols_1<N1, N2><<<dim3(M / kCols, N2), Plan<N1>::T * kCols, 0, st>>>(tmp, tw1, wm, ds);
    k_fft_cols_2<N1, N2><<<dim3(M / kCols, N1), Plan<N2>::T * kCols, 0, st>>>(tmp, out, tw2, ds);
    return cudaGetLastError();
}

cudaError_t fft2d_large(const float2* in, float2* out, float2* tmp, int M, int sign, cudaStream_t st)
{
    if (M == 4096) return fft2d_large_t<64, 64>(in, out, tmp, sign, st);
    if (M == 8192) return fft2d_large_t<64, 128>(in, out, tmp, sign, st);
    return cudaErrorInvalidValue;
}

}  // namespace atmwfs
