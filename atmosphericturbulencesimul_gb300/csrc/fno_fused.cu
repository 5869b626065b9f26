// fno_fused.cu -- the surrogate's default shape (grid 256, 32 modes, width 64,
// projection 128) as kernels that fuse neighbouring products on the tcgen05
// tensor cores, so that the images between them are not written and read
// back:
//   k_xdft     the forward DFT along x, written as coalesced spectrum rows
//              (of the lift's output, for a number of input planes other than 8);
//   k_yfwd, k_yinv  the DFTs along y;
//   k_fourier  pointwise mixing + inverse DFT along x (+ bias, GELU, and the
//              next layer's forward DFT along x), the lift with its DFT, and
//              the same pair of the backward pass;
//   k_project  the first projection + GELU + the 2-channel output;
//   k_layer_bwd  a layer's GELU gradient, its weight and bias gradients and
//              the transposed inverse DFT along x, from one read of the line;
//   k_project_bwd  every gradient of the head, without storing dq.
// The products keep the operands' BF16 rounding and the FP32 accumulation of the
// separate products (k_pointwise, k_rowprod, the mma.sync GEMM).  The order of
// the additions is not the same everywhere (the head's two outputs, sums over
// pixels), so results agree to FP32 rounding, not in every bit: outputs to 2e-7 of
// their scale with the tcgen05 products.
//
// Spectral images here are planar with the channels fastest, so that a
// mode's values of every channel are one run (the mode mixing) and a
// warp's channels store as one (k_xdft): with BW = B w,
//   a, bb : [2][G][m][BW]  (real / imaginary plane, row y, kx, channel)
//   z, y  : [2 m][m][BW]   (row ky: real parts, row m + ky: imaginary parts)
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "atmwfs_fno.h"
#include "fno_gemm.cuh"
#include "umma_core.cuh"

namespace atmwfs {
namespace umma {

constexpr int kG = 256;       // grid side
constexpr int kModes = 32;    // modes per axis
constexpr int kW = 64;        // width
constexpr int kProj = 128;    // projection channels
constexpr long kP = (long)kG * kG;

__device__ __forceinline__ uint4 pack8(const float (&f)[8])
{
    __nv_bfloat162 h[4];
#pragma unroll
    for (int q = 0; q < 4; q++) h[q] = __floats2bfloat162_rn(f[2 * q], f[2 * q + 1]);
    uint4 v;
    v.x = *reinterpret_cast<uint32_t*>(&h[0]);
    v.y = *reinterpret_cast<uint32_t*>(&h[1]);
    v.z = *reinterpret_cast<uint32_t*>(&h[2]);
    v.w = *reinterpret_cast<uint32_t*>(&h[3]);
    return v;
}

// ---------------------------------------------------------------------------
// Forward DFT along x of one line (sample b, row y), all channels:
//   a[p][y][kx][b w + c] = sum_x h[b][c][y][x] F[p m + kx][x]
// as D = h F^T: the 64 channels are the MMA's M (rows 64 .. 127 of the 128 are
// whatever follows in shared memory, here F, and their results are not read),
// the 64 rows of F its N, K = 256.  With the channels along the TMEM lanes a
// mode's values leave as one 128-byte run per warp.  (k_rowprod has the lines
// of all channels along the lanes and writes 16-byte pieces 128 bytes apart:
// the rate of L2 requests bounds it, 138 us for a batch of 16 against 49 us of
// HBM time; this form takes 57 us.)
// F is staged once per CTA; a line's 64 KB are loaded into registers while the
// previous line's products run, so a CTA keeps 64 KB in flight.
// ---------------------------------------------------------------------------
constexpr int kXK = kG / 8;                        // core matrices along K
constexpr uint32_t kXBytes = 2 * kModes * kG * 2;  // F, and one line of 64 channels, in BF16: 32 KB each
static_assert(2 * kModes == kW, "the two operands have the same shape");

// piece j of thread tid: 8 consecutive x of one channel; the lanes of a warp
// take 8 channels x 4 pieces, so that a store phase of 8 lanes fills one
// 128-byte core matrix
template <int NT = kThreads>
__device__ __forceinline__ void x_piece(int tid, int j, int& row, int& k8)
{
    const int i = tid + NT * j, rest = i >> 5;
    row = (rest & 7) * 8 + (i & 7);
    k8 = (rest >> 3) * 4 + ((i >> 3) & 3);
}

// The 64 x 64 spectrum of a line from tensor memory (lanes 0 .. 63: channels,
// columns: re and im of the modes) into the planar image, by the warps of the
// lower two lane blocks: warp w takes lanes 32 (w % 4) .. and the w / 4-th of
// S equal ranges of columns.
template <int S>
__device__ __forceinline__ void store_spectrum(uint32_t tmem, float* __restrict__ a, int line, long Nc, int warp, int lane)
{
    const int cb = (warp & 3) * 32, b = line / kG, y = line % kG;
    const size_t BW = (size_t)Nc / kModes;
#pragma unroll
    for (int c0 = 0; c0 < kW / S; c0 += 16) {
        const int n = (warp >> 2) * (kW / S) + c0, p = n / kModes, kx = n % kModes;
        float* o = a + (size_t)p * kG * Nc + (size_t)y * Nc + kx * BW + (size_t)b * kW + cb + lane;
        float r[16];
        tmem_ld16(tmem + ((uint32_t)cb << 16) + n, r);
#pragma unroll
        for (int q = 0; q < 16; q++) o[q * BW] = r[q];
    }
}

__global__ void __launch_bounds__(kThreads, 2) k_xdft(const __nv_bfloat16* __restrict__ F, const float* __restrict__ H,
                                                      float* __restrict__ a, int nlines, long Nc, unsigned* status)
{
    constexpr int J = kW * kXK / kThreads;  // pieces per thread
    extern __shared__ __align__(128) unsigned char sm[];
    unsigned char *sa = sm, *sb = sm + kXBytes;  // the line, F
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float4 v[J][2];
    auto load = [&](int line, int j) {
        int row, k8;
        x_piece(tid, j, row, k8);
        const float4* q = reinterpret_cast<const float4*>(H + (size_t)(line / kG) * kW * kP + (size_t)(line % kG) * kG +
                                                          (size_t)row * kP + k8 * 8);
        v[j][0] = __ldg(q);
        v[j][1] = __ldg(q + 1);
    };
    if (blockIdx.x < nlines)
#pragma unroll
        for (int j = 0; j < J; j++) load(blockIdx.x, j);
    tmem_alloc(&tmem_base, 64, warp);
    if (tid == 0) mbar_init(&bar);
#pragma unroll
    for (int j = 0; j < J; j++) {
        int row, k8;
        x_piece(tid, j, row, k8);
        *reinterpret_cast<uint4*>(sb + kmajor_off(row, k8 * 8, kXK)) =
            *reinterpret_cast<const uint4*>(F + (size_t)row * kG + k8 * 8);
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_base, a_addr = smem_addr(sa), b_addr = smem_addr(sb);
    uint32_t parity = 0;
    for (int line = blockIdx.x; line < nlines; line += gridDim.x) {
#pragma unroll
        for (int j = 0; j < J; j++) {
            int row, k8;
            x_piece(tid, j, row, k8);
            const float f[8] = {v[j][0].x, v[j][0].y, v[j][0].z, v[j][0].w, v[j][1].x, v[j][1].y, v[j][1].z, v[j][1].w};
            *reinterpret_cast<uint4*>(sa + kmajor_off(row, k8 * 8, kXK)) = pack8(f);
            if (line + (int)gridDim.x < nlines) load(line + gridDim.x, j);
        }
        publish_smem();
        if (tid == 0) {
#pragma unroll
            for (int ks = 0; ks < kG / 16; ks++)
                mma_bf16(tmem, smem_desc(a_addr + ks * 256, 128, kXK * 128), smem_desc(b_addr + ks * 256, 128, kXK * 128),
                         instr_desc(kW), ks > 0);
            mma_commit(&bar);
        }
        if (!mma_wait(&bar, parity, status)) break;
        parity ^= 1;
        if ((warp & 3) < 2) store_spectrum<2>(tmem, a, line, Nc, warp, lane);
        retire_tile();
    }
    tmem_free(tmem, 64, warp);
}

// ---------------------------------------------------------------------------
// The DFTs along y over the P = m B w columns of the planar images:
//   k_yfwd  z (64 x P) = F (64 x 512) a (512 x P)     (64 rows: re, im of the kept ky)
//   k_yinv  bb (512 x P) = G (512 x 64) y (64 x P)
// 128 columns per tile along the TMEM lanes.  An image is 67 MB at a batch of 16
// (10 us of HBM time, or L2): latency is what has to be hidden.  k_yfwd takes
// K in four chunks of 128 whose next values are loaded into registers as the
// current ones are stored (eight staged chunks of 64 before: 31-33 us).  k_yinv
// gives each CTA a quarter of the output rows, so that four CTAs share an SM
// and its 512 columns of tensor memory (one CTA per SM held all 512 rows
// before, 256 tiles on 152 CTAs: 31 us).
// The backward pass has the same two: dy = GyBig^T dbb, da = FyAB^T dz, and
// GyBig^T is FyAB, value by value.  SPLIT (dy) keeps a chunk's products in an
// accumulator of their own and adds the four in FP32, as the split product
// did that this replaces (K = 128 per run, four atomic adds into a cleared dy:
// 45 us for a batch of 8, now 21).
// ---------------------------------------------------------------------------
constexpr int kYK = 2 * kG;                      // K of the forward product
constexpr int kYC = 128;                         // its chunk
constexpr uint32_t kYA = 2 * kModes * kYK * 2;   // F: 64 KB, then the chunk's A tile: 32 KB
constexpr uint32_t kYBytes = kYA + kM * kYC * 2;

template <bool SPLIT>
__global__ void __launch_bounds__(kThreads, 2) k_yfwd(const __nv_bfloat16* __restrict__ F, const float* __restrict__ X,
                                                      float* __restrict__ Z, long P, int ntiles, unsigned* status)
{
    constexpr int J = kYC / 16;       // pieces of 8 rows per thread
    constexpr int NC = kYK / kYC;
    constexpr int NA = SPLIT ? NC : 1;  // accumulators, 64 columns each
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m = tid % kM, kc0 = tid / kM;
    float x[J][8];
    auto load = [&](int tile, int chunk, int j) {
        const float* src = X + (size_t)(chunk * kYC + (kc0 + 2 * j) * 8) * P + (size_t)tile * kM + m;
#pragma unroll
        for (int q = 0; q < 8; q++) x[j][q] = __ldg(src + (size_t)q * P);
    };
    if (blockIdx.x < ntiles)
#pragma unroll
        for (int j = 0; j < J; j++) load(blockIdx.x, 0, j);
    tmem_alloc(&tmem_base, 64 * NA, warp);
    if (tid == 0) mbar_init(&bar);
    for (int i = tid; i < 2 * kModes * kYK / 8; i += kThreads) {
        const int row = (i >> 9) * 8 + (i & 7), k8 = (i >> 3) & 63;
        *reinterpret_cast<uint4*>(sm + kmajor_off(row, k8 * 8, kYK / 8)) =
            *reinterpret_cast<const uint4*>(F + (size_t)row * kYK + k8 * 8);
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_base, base = smem_addr(sm);
    uint32_t parity = 0;
    bool failed = false;
    for (int tile = blockIdx.x; tile < ntiles && !failed; tile += gridDim.x) {
#pragma unroll 1
        for (int c = 0; c < NC; c++) {
            const bool more = c + 1 < NC || tile + (int)gridDim.x < ntiles;
            const int nt = c + 1 < NC ? tile : tile + gridDim.x, nc = c + 1 < NC ? c + 1 : 0;
#pragma unroll
            for (int j = 0; j < J; j++) {
                *reinterpret_cast<uint4*>(sm + kYA + kmajor_off(m, (kc0 + 2 * j) * 8, kYC / 8)) = pack8(x[j]);
                if (more) load(nt, nc, j);
            }
            publish_smem();
            if (tid == 0) {
#pragma unroll
                for (int ks = 0; ks < kYC / 16; ks++)
                    mma_bf16(tmem + (SPLIT ? c * 64 : 0), smem_desc(base + kYA + ks * 256, 128, kYC / 8 * 128),
                             smem_desc(base + c * (kYC / 8) * 128 + ks * 256, 128, kYK / 8 * 128), instr_desc(2 * kModes),
                             (!SPLIT && c > 0) || ks > 0);
                mma_commit(&bar);
            }
            // the chunk's products are done before its A tile is overwritten
            if (!mma_wait(&bar, parity, status)) {
                failed = true;
                break;
            }
            parity ^= 1;
        }
        if (failed) break;
        const int g = warp & 3, half = warp >> 2;
        float* o = Z + (size_t)tile * kM + g * 32 + lane;
#pragma unroll
        for (int c0 = half * kModes; c0 < (half + 1) * kModes; c0 += 16) {
            float r[16];
            tmem_ld16(tmem + ((uint32_t)(g * 32) << 16) + c0, r);
#pragma unroll
            for (int p = 1; p < NA; p++) {
                float t[16];
                tmem_ld16(tmem + ((uint32_t)(g * 32) << 16) + p * 64 + c0, t);
#pragma unroll
                for (int q = 0; q < 16; q++) r[q] += t[q];
            }
#pragma unroll
            for (int q = 0; q < 16; q++) o[(size_t)(c0 + q) * P] = r[q];
        }
        retire_tile();
    }
    tmem_free(tmem, 64 * NA, warp);
}

constexpr int kYQ = kYK / 4;                              // output rows per CTA
constexpr uint32_t kIA = kYQ * 2 * kModes * 2;            // its rows of G: 16 KB, then the A tile: 16 KB
constexpr uint32_t kIBytes = kIA + kM * 2 * kModes * 2;

__global__ void __launch_bounds__(kThreads, 4) k_yinv(const __nv_bfloat16* __restrict__ Gy, const float* __restrict__ X,
                                                      float* __restrict__ bb, long P, int ntiles, unsigned* status)
{
    constexpr int K = 2 * kModes, J = K / 16;
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m = tid % kM, kc0 = tid / kM;
    const int quarter = blockIdx.x & 3, step = gridDim.x >> 2;
    float x[J][8];
    auto load = [&](int tile, int j) {
        const float* src = X + (size_t)((kc0 + 2 * j) * 8) * P + (size_t)tile * kM + m;
#pragma unroll
        for (int q = 0; q < 8; q++) x[j][q] = __ldg(src + (size_t)q * P);
    };
    const int first = blockIdx.x >> 2;
    if (first < ntiles)
#pragma unroll
        for (int j = 0; j < J; j++) load(first, j);
    tmem_alloc(&tmem_base, kYQ, warp);
    if (tid == 0) mbar_init(&bar);
    for (int i = tid; i < kYQ * K / 8; i += kThreads) {
        const int row = (i >> 6) * 8 + (i & 7), k8 = (i >> 3) & 7;
        *reinterpret_cast<uint4*>(sm + kmajor_off(row, k8 * 8, K / 8)) =
            *reinterpret_cast<const uint4*>(Gy + (size_t)(quarter * kYQ + row) * K + k8 * 8);
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_base, base = smem_addr(sm);
    uint32_t parity = 0;
    for (int tile = first; tile < ntiles; tile += step) {
#pragma unroll
        for (int j = 0; j < J; j++) {
            *reinterpret_cast<uint4*>(sm + kIA + kmajor_off(m, (kc0 + 2 * j) * 8, K / 8)) = pack8(x[j]);
            if (tile + step < ntiles) load(tile + step, j);
        }
        publish_smem();
        if (tid == 0) {
#pragma unroll
            for (int ks = 0; ks < K / 16; ks++)
                mma_bf16(tmem, smem_desc(base + kIA + ks * 256, 128, K / 8 * 128), smem_desc(base + ks * 256, 128, K / 8 * 128),
                         instr_desc(kYQ), ks > 0);
            mma_commit(&bar);
        }
        if (!mma_wait(&bar, parity, status)) break;
        parity ^= 1;
        const int g = warp & 3, half = warp >> 2;
        float* o = bb + (size_t)quarter * kYQ * P + (size_t)tile * kM + g * 32 + lane;
#pragma unroll 1
        for (int c0 = half * (kYQ / 2); c0 < (half + 1) * (kYQ / 2); c0 += 16) {
            float r[16];
            tmem_ld16(tmem + ((uint32_t)(g * 32) << 16) + c0, r);
#pragma unroll
            for (int q = 0; q < 16; q++) o[(size_t)(c0 + q) * P] = r[q];
        }
        retire_tile();
    }
    tmem_free(tmem, kYQ, warp);
}

// ---------------------------------------------------------------------------
// A Fourier layer's output u = W h + b + S, S the inverse DFT along x of the
// planar spectrum bb, and act = gelu(u): for 128 pixels of a line (sample b,
// row y, half of x)
//   D1 = X^T W^T   (128 pixels x 64 channels, K = 64 channels)
//   D2 = Gx^T B^T  (128 pixels x 64 channels, K = 64: re and im of 32 modes)
// in two ranges of tensor memory, added in the epilogue in the order of the
// separate products.  The inverse DFT's image is 268 MB per layer and batch
// of 16: it was written in 16-byte pieces (126 us) and read back by the
// pointwise product (161 us); both now run as one pass over h and bb.
// Gx^T and W are staged once per CTA; a tile's 32 channel values per thread
// and the line's spectrum are loaded while the previous tile's products run.
// The backward pass of a layer ends with the same pair: dh = W^T du + Fx da
// (TW: W transposed; Gt = Fx; no bias).
//
// DFT: the next layer's forward DFT along x, from the same registers:
//   D3 = act F^T   (64 channels x 64, K = 256 x, half a line per tile)
// The epilogue leaves the tile's BF16 values in shared memory (two pixels of
// a channel per word: neighbouring lanes trade one value), their products are
// issued with the next tile's and the line's spectrum is stored after them, so
// that nothing more is waited for.  At a batch of 16, k_fourier 137 us and a
// k_xdft of 76 us (which read 268 MB again) became 168 us; the lift, 72 us
// and 76, became 70 us.  The bias is read from shared memory: the tiles take
// the L1 that the operands leave (28 KB), so each read of the global array went
// to L2 (193 us).
// KX = 8 without SPEC is the lift (K padded to 16 with zero channels; no
// activation).
// ---------------------------------------------------------------------------
constexpr int kFK = kW / 8;  // core matrices along a K of 64

// A stored pixel pair is one word per lane: 8-pixel groups 1056 bytes apart
// put a warp's four groups x two channels into all 32 banks.
constexpr uint32_t kHL = kW / 8 * 128 + 32;
__device__ __forceinline__ uint32_t h_off(int ch, int px)
{
    return (uint32_t)((px >> 3) * kHL + (ch >> 3) * 128 + (ch & 7) * 16 + (px & 7) * 2);
}

// shared-memory offsets: W, Gt, the tile's X, the line's spectrum, then the
// tile's outputs (whose MMA rows 64 .. 127 read on into F) and F
template <bool SPEC, int KX, bool DFT>
struct FourierSmem {
    static constexpr int K = KX < 16 ? 16 : KX, KC = K / 8;
    static constexpr uint32_t w = 0, g = w + kW * K * 2, x = g + (SPEC ? kG * kW * 2 : 0), s = x + kM * K * 2,
                              h = s + (SPEC ? kW * kW * 2 : 0), f = h + (DFT ? kM / 8 * kHL : 0),
                              bytes = f + (DFT ? kXBytes : 0);
};

template <bool TW, bool SPEC, int KX, bool DFT>
__global__ void __launch_bounds__(kThreads, SPEC ? 2 : 3)
    k_fourier(const __nv_bfloat16* __restrict__ W, const __nv_bfloat16* __restrict__ Gt, const float* __restrict__ X,
              const float* __restrict__ bb, float* __restrict__ U, float* __restrict__ act,
              const float* __restrict__ bias, const __nv_bfloat16* __restrict__ F, float* __restrict__ a, int nlines,
              long Nc, unsigned* status, int write_u)
{
    using S = FourierSmem<SPEC, KX, DFT>;
    constexpr int KC = S::KC, J = S::K / 16, GC = kFK;
    constexpr uint32_t kD3 = SPEC ? 2 * kW : kW, kCols = DFT && SPEC ? 256 : 128;
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base;
    __shared__ float s_bias[kW];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m = tid % kM, kc0 = tid / kM;  // this thread's pixel and first channel group (of 8): kc0, kc0 + 2, ...
    const int so = tid & 63, sk = tid >> 6;  // its spectrum channel, and mode groups (of 8) sk, sk + 4
    const size_t BW = (size_t)Nc / kModes;
    float x[J][8], s[2][8];
    auto load_x = [&](int line, int half) {
        const float* src = X + (size_t)(line / kG) * KX * kP + (size_t)(line % kG) * kG + half * kM + m;
#pragma unroll
        for (int j = 0; j < J; j++)
#pragma unroll
            for (int q = 0; q < 8; q++)
                x[j][q] = KX >= 16 || kc0 == 0 ? __ldg(src + (size_t)((kc0 + 2 * j) * 8 + q) * kP) : 0.0f;
    };
    auto load_s = [&](int line) {
        if (!SPEC) return;
        const float* src = bb + (size_t)(line % kG) * Nc + (size_t)sk * 8 * BW + (size_t)(line / kG) * kW + so;
#pragma unroll
        for (int j = 0; j < 2; j++)  // j: real, imaginary plane
#pragma unroll
            for (int q = 0; q < 8; q++) s[j][q] = __ldg(src + (size_t)j * kG * Nc + q * BW);
    };
    if (blockIdx.x < nlines) {
        load_x(blockIdx.x, 0);
        load_s(blockIdx.x);
    }
    tmem_alloc(&tmem_base, kCols, warp);
    if (tid == 0) mbar_init(&bar);
    if (tid < kW) s_bias[tid] = bias ? bias[tid] : 0.0f;
    // the weights: element loads (a parameter block carries no alignment guarantee)
    for (int i = tid; i < kW * S::K; i += kThreads) {
        const int row = i / S::K, k = i % S::K;  // TW: of W^T
        *reinterpret_cast<__nv_bfloat16*>(sm + S::w + kmajor_off(TW ? k : row, TW ? row : k, KC)) =
            k < KX ? W[row * KX + k] : __float2bfloat16_rn(0.0f);
    }
    if (SPEC)
        for (int i = tid; i < kG * GC; i += kThreads) {
            const int row = (i >> 6) * 8 + (i & 7), k8 = (i >> 3) & 7;
            *reinterpret_cast<uint4*>(sm + S::g + kmajor_off(row, k8 * 8, GC)) =
                *reinterpret_cast<const uint4*>(Gt + (size_t)row * kW + k8 * 8);
        }
    if (DFT)
        for (int i = tid; i < 2 * kModes * kXK; i += kThreads) {
            int row, k8;
            x_piece(tid, i / kThreads, row, k8);
            *reinterpret_cast<uint4*>(sm + S::f + kmajor_off(row, k8 * 8, kXK)) =
                *reinterpret_cast<const uint4*>(F + (size_t)row * kG + k8 * 8);
        }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_base, base = smem_addr(sm);
    // the products of the last tile's outputs, K = its half of x (one thread issues)
    auto dft = [&](int half) {
#pragma unroll
        for (int ks = 0; ks < kM / 16; ks++)
            mma_bf16(tmem + kD3, smem_desc(base + S::h + ks * 2 * kHL, kHL, 128),
                     smem_desc(base + S::f + half * (kM / 8) * 128 + ks * 256, 128, kXK * 128), instr_desc(kW),
                     half > 0 || ks > 0);
    };
    uint32_t parity = 0;
    bool failed = false;
    int last = -1;  // the line whose second half is in shared memory
    const int ntiles = 2 * nlines;
    // tiles in pairs: both halves of a line, then the CTA's next line
    for (int tile = 2 * blockIdx.x; tile < ntiles; tile += (tile & 1) ? 2 * (int)gridDim.x - 1 : 1) {
        const int line = tile >> 1, half = tile & 1;
#pragma unroll
        for (int j = 0; j < J; j++)
            *reinterpret_cast<uint4*>(sm + S::x + kmajor_off(m, (kc0 + 2 * j) * 8, KC)) = pack8(x[j]);
        if (SPEC && half == 0) {
#pragma unroll
            for (int j = 0; j < 2; j++)
                *reinterpret_cast<uint4*>(sm + S::s + kmajor_off(so, (sk + 4 * j) * 8, GC)) = pack8(s[j]);
        }
        publish_smem();
        if (half == 0) {
            load_x(line, 1);
        } else if (line + (int)gridDim.x < nlines) {
            load_x(line + gridDim.x, 0);
            load_s(line + gridDim.x);
        }
        if (tid == 0) {
#pragma unroll
            for (int ks = 0; ks < S::K / 16; ks++)
                mma_bf16(tmem, smem_desc(base + S::x + ks * 256, 128, KC * 128),
                         smem_desc(base + S::w + ks * 256, 128, KC * 128), instr_desc(kW), ks > 0);
            if (SPEC) {
#pragma unroll
                for (int ks = 0; ks < kW / 16; ks++)
                    mma_bf16(tmem + kW, smem_desc(base + S::g + half * (kM / 8) * GC * 128 + ks * 256, 128, GC * 128),
                             smem_desc(base + S::s + ks * 256, 128, GC * 128), instr_desc(kW), ks > 0);
            }
            if (DFT && (half == 1 || last >= 0)) dft(half ^ 1);
            mma_commit(&bar);
        }
        if (!mma_wait(&bar, parity, status)) {
            failed = true;
            break;
        }
        parity ^= 1;
        if (DFT && half == 0 && last >= 0 && (warp & 3) < 2) store_spectrum<2>(tmem + kD3, a, last, Nc, warp, lane);
        const int g = warp & 3, ch = warp >> 2;
        const uint32_t trow = tmem + ((uint32_t)(g * 32) << 16);
        const size_t o0 = (size_t)(line / kG) * kW * kP + (size_t)(line % kG) * kG + half * kM + g * 32 + lane;
#pragma unroll 1
        for (int c0 = ch * (kW / 2); c0 < (ch + 1) * (kW / 2); c0 += 16) {
            float r[16], sp[16];
            tmem_ld16(trow + c0, r);
            if (SPEC) tmem_ld16(trow + kW + c0, sp);
#pragma unroll
            for (int q = 0; q < 16; q++) {
                const size_t o = o0 + (size_t)(c0 + q) * kP;
                float u = r[q] + s_bias[c0 + q];
                if (SPEC) u += sp[q];
                if (write_u) U[o] = u;
                if (SPEC && act) act[o] = u = gelu_f(u);
                r[q] = u;
            }
            if (DFT) {
                const bool odd = lane & 1;
#pragma unroll
                for (int q = 0; q < 16; q += 2) {  // even lanes: channel q, odd lanes: q + 1; pixels lane & ~1, + 1
                    const float other = __shfl_xor_sync(0xFFFFFFFFu, odd ? r[q] : r[q + 1], 1);
                    *reinterpret_cast<__nv_bfloat162*>(sm + S::h + h_off(c0 + q + odd, g * 32 + (lane & ~1))) =
                        __floats2bfloat162_rn(odd ? other : r[q], odd ? r[q + 1] : other);
                }
            }
        }
        if (half == 1) last = line;
        retire_tile();
    }
    if (DFT && !failed && last >= 0) {  // the CTA's last line
        publish_smem();
        if (tid == 0) {
            dft(1);
            mma_commit(&bar);
        }
        if (mma_wait(&bar, parity, status) && (warp & 3) < 2) store_spectrum<2>(tmem + kD3, a, last, Nc, warp, lane);
        fence_before();
    }
    tmem_free(tmem, kCols, warp);
}

// ---------------------------------------------------------------------------
// A layer's backward products over one line (sample b, row y), from one read
// of dh, u and h:
//   du = dh gelu'(u)                              (ACT; else du = dh, not written)
//   dbb = the transposed inverse DFT along x: D1 = du Gx^T (64 channels x 64, K = 256 x)
//   dW += du h^T                              D2 (64 x 64, K = 256 x, over lines)
//   db += sum_x du
// HBM bounds it: 0.57 GB for a batch of 8.  As separate kernels the gradient
// (74 us), the weight product (93), the bias sums (37) and the DFT (67) read du
// three times more.  The line's du is the A operand of both products (rows 64
// .. 127 of the MMA's M are what follows in shared memory and are not read);
// D2 stays in tensor memory for kFlush lines (K = 1024, the longest run of the
// split product it replaces) and is then added to FP32 registers, one atomic
// per element and CTA at the end.
// db (and the head's sums over pixels, below): a line's values are added in
// FP32, the lines to a pair in shared memory (the registers are taken) and the
// CTAs' totals in FP64, 2^-24 of the sum in all.  One FP32 register per thread
// for all lines and FP32 atomics of 152 CTAs were twice as far from the exact
// sums as k_rowsum's 64 CTAs (up to 22 times for dc2); FP64 additions per line
// would share the part's few FP64 lanes with nothing to gain.
// ---------------------------------------------------------------------------
// HC = 8 without SPEC is the lift's weight and bias gradient (no DFT, K the
// input planes padded to 16 zero rows).
//
// One CTA of 512 threads per SM: a line's operands (up to 192 KB) are loaded
// into registers, each piece as soon as the previous line's is used.
constexpr int kFlush = 4;
constexpr int kBT = 512;

__device__ __forceinline__ void ld8(float (&f)[8], const float* p)
{
    const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
    f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}

// A thread's sum over lines as hi + lo; an overflowed or undefined hi is the value.
__device__ __forceinline__ void pair_add(float2& s, float v)
{
    const float t = s.x + v, b = t - s.x;
    s.y += (s.x - (t - b)) + (v - b);
    s.x = t;
}
__device__ __forceinline__ double pair_value(float2 s)
{
    return fabsf(s.x) <= FLT_MAX ? (double)s.x + (double)s.y : (double)s.x;
}
__device__ __forceinline__ float sum8(const float (&f)[8])
{
    return ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]));
}

constexpr uint32_t kLBytes = 3 * kXBytes + kBT * 8;  // du, Gx, h, the threads' bias sums

template <bool ACT, bool SPEC, int HC>
__global__ void __launch_bounds__(kBT, 1)
    k_layer_bwd(const __nv_bfloat16* __restrict__ Gx, const float* __restrict__ dh, const float* __restrict__ u,
                const float* __restrict__ h, float* __restrict__ du, float* __restrict__ dbb, float* __restrict__ dW,
                double* __restrict__ db, int nlines, long Nc, unsigned* status)
{
    constexpr int J = kW * kXK / kBT;            // pieces of the line per thread
    constexpr int HN = HC < 16 ? 16 : HC;        // N of the weight product
    constexpr int JH = HC == kW ? J : 1;         // pieces of h per thread
    constexpr int CN = HN / 4;                   // dW columns per reading thread (4 warps per lane block)
    static_assert(HC == kW || HC * kXK <= kBT, "h in one piece per thread");
    extern __shared__ __align__(128) unsigned char sm[];
    unsigned char *sd = sm, *sg = sm + kXBytes, *sh = sm + 2 * kXBytes;  // du, Gx, h
    float2& bsum = reinterpret_cast<float2*>(sm + 3 * kXBytes)[threadIdx.x];  // every piece of a thread has the same channel
    bsum = make_float2(0.0f, 0.0f);
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float d[J][8], g[ACT ? J : 1][8], hv[JH][8];
    const int hrow = tid & 7, hk8 = tid >> 3;    // HC = 8: this thread's piece of h
    auto load = [&](int line, int j) {
        const size_t o0 = (size_t)(line / kG) * kW * kP + (size_t)(line % kG) * kG;
        int row, k8;
        x_piece<kBT>(tid, j, row, k8);
        const size_t o = o0 + (size_t)row * kP + k8 * 8;
        ld8(d[j], dh + o);
        if constexpr (ACT) ld8(g[j], u + o);
        if constexpr (HC == kW) ld8(hv[j], h + o);
    };
    auto load_h = [&](int line) {
        if constexpr (HC != kW)
            if (tid < HC * kXK)
                ld8(hv[0], h + (size_t)(line / kG) * HC * kP + (size_t)(line % kG) * kG + (size_t)hrow * kP + hk8 * 8);
    };
    if (blockIdx.x < nlines) {
#pragma unroll
        for (int j = 0; j < J; j++) load(blockIdx.x, j);
        load_h(blockIdx.x);
    }
    tmem_alloc(&tmem_base, 128, warp);
    if (tid == 0) mbar_init(&bar);
    if constexpr (SPEC) {
#pragma unroll
        for (int j = 0; j < J; j++) {
            int row, k8;
            x_piece<kBT>(tid, j, row, k8);
            *reinterpret_cast<uint4*>(sg + kmajor_off(row, k8 * 8, kXK)) =
                *reinterpret_cast<const uint4*>(Gx + (size_t)row * kG + k8 * 8);
        }
    }
    if constexpr (HC != kW) {
        static_assert(HC == kW || HC == 8, "one group of valid rows, one of zeros");
        if (tid < 8 * kXK)
            *reinterpret_cast<uint4*>(sh + kmajor_off(8 + hrow, hk8 * 8, kXK)) = make_uint4(0u, 0u, 0u, 0u);
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_base, d_addr = smem_addr(sd), g_addr = smem_addr(sg), h_addr = smem_addr(sh);
    uint32_t parity = 0;
    float acc[CN];      // dW of o = the lane's channel: the warps that read tensor memory
#pragma unroll
    for (int q = 0; q < CN; q++) acc[q] = 0.0f;
    const bool reads = (warp & 3) < 2;
    const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    int held = 0;  // lines in D2
    for (int line = blockIdx.x; line < nlines; line += gridDim.x) {
        const size_t o0 = (size_t)(line / kG) * kW * kP + (size_t)(line % kG) * kG;
        float ls = 0.0f;
#pragma unroll
        for (int j = 0; j < J; j++) {
            int row, k8;
            x_piece<kBT>(tid, j, row, k8);
            if constexpr (ACT) {
#pragma unroll
                for (int q = 0; q < 8; q++) d[j][q] *= gelu_d(g[j][q]);
                float4* o = reinterpret_cast<float4*>(du + o0 + (size_t)row * kP + k8 * 8);
                o[0] = make_float4(d[j][0], d[j][1], d[j][2], d[j][3]);
                o[1] = make_float4(d[j][4], d[j][5], d[j][6], d[j][7]);
            }
            ls += sum8(d[j]);
            *reinterpret_cast<uint4*>(sd + kmajor_off(row, k8 * 8, kXK)) = pack8(d[j]);
            if constexpr (HC == kW) *reinterpret_cast<uint4*>(sh + kmajor_off(row, k8 * 8, kXK)) = pack8(hv[j]);
            // the piece's registers are free: the next line's values come in
            // under the remaining pieces' arithmetic and the products
            if (line + (int)gridDim.x < nlines) load(line + gridDim.x, j);
        }
        pair_add(bsum, ls);
        if constexpr (HC != kW)
            if (tid < HC * kXK) *reinterpret_cast<uint4*>(sh + kmajor_off(hrow, hk8 * 8, kXK)) = pack8(hv[0]);
        if (line + (int)gridDim.x < nlines) load_h(line + gridDim.x);
        publish_smem();
        if (tid == 0) {
#pragma unroll
            for (int ks = 0; ks < kG / 16; ks++) {
                const uint64_t da = smem_desc(d_addr + ks * 256, 128, kXK * 128);
                if constexpr (SPEC)
                    mma_bf16(tmem, da, smem_desc(g_addr + ks * 256, 128, kXK * 128), instr_desc(kW), ks > 0);
                mma_bf16(tmem + kW, da, smem_desc(h_addr + ks * 256, 128, kXK * 128), instr_desc(HN), ks > 0 || held > 0);
            }
            mma_commit(&bar);
        }
        if (!mma_wait(&bar, parity, status)) break;
        parity ^= 1;
        const bool flush = ++held == kFlush || line + (int)gridDim.x >= nlines;
        if (reads) {
            if constexpr (SPEC) store_spectrum<4>(tmem, dbb, line, Nc, warp, lane);
            if (flush) {
                float r[16];
                tmem_ld16(trow + kW + (HN == 16 ? 0 : (warp >> 2) * CN), r);
                if constexpr (HN == 16) {
#pragma unroll
                    for (int q = 0; q < CN; q++) acc[q] += (warp >> 2) < 2 ? r[((warp >> 2) & 1) * CN + q] : 0.0f;
                } else {
#pragma unroll
                    for (int q = 0; q < CN; q++) acc[q] += r[q];
                }
            }
        }
        if (flush) held = 0;
        retire_tile();
    }
    if (reads && (warp >> 2) * CN < HC) {
        float* o = dW + ((warp & 3) * 32 + lane) * HC + (warp >> 2) * CN;
#pragma unroll
        for (int q = 0; q < CN; q++) atomicAdd(o + q, acc[q]);
    }
    // a channel's lanes: l, l + 8, l + 16, l + 24 of warps w and w + 8
    double bs = pair_value(bsum);
    bs += __shfl_xor_sync(0xffffffffu, bs, 8);
    bs += __shfl_xor_sync(0xffffffffu, bs, 16);
    if (lane < 8) atomicAdd(db + (warp & 7) * 8 + lane, bs);
    tmem_free(tmem, 128, warp);
}

// ---------------------------------------------------------------------------
// Backward of the projection head over one line (sample b, row y):
//   dq = (W2^T dout) gelu'(qpre)         (128 channels)
//   dh = W1^T dq                         D3 (256 pixels x 64 channels, K = 128)
//   dW1 += dq u^T, dc1 += sum dq         D2 (128 x 64, K = 256 pixels, over lines)
//   dW2 += dout q^T, dc2 += sum dout     q = gelu(qpre), from the same tanh
// from one read of qpre, u and dout; dq stays on the SM (as BF16, as every
// product rounds it; its bias sums are FP32).  HBM bounds it: 0.54 GB for a
// batch of 8.  Before: a GEMM of K = 2 writing dq (129 us), its GELU gradient
// (120), three products reading dq or q (104 + 130 + 244) and the bias sums
// (75).  dq is stored twice in shared memory, [channel][pixel] for dW1 and
// [pixel][channel] for dh (each K-major); the second's 8-row groups are 32
// bytes apart from a multiple of 128 so that its 2-byte stores spread over the
// banks.
// ---------------------------------------------------------------------------
constexpr uint32_t kQA = 0;                                   // dq [128][256 px]
constexpr uint32_t kQU = kQA + kProj * kG * 2;                // u [64][256 px]
constexpr uint32_t kQTs = kProj / 8 * 128 + 32;               // bytes between 8-pixel groups of dq^T
constexpr uint32_t kQT = kQU + kW * kG * 2;                   // dq^T [256 px][128]
constexpr uint32_t kQW = kQT + kG / 8 * kQTs;                 // W1^T [64][128]
constexpr uint32_t kQS = kQW + kW * kProj * 2;                // the threads' sums: dc1 and dW2 of two channels, dc2
constexpr int kQSums = 7;
constexpr uint32_t kQBytes = kQS + kQSums * kBT * 8;

__global__ void __launch_bounds__(kBT, 1)
    k_project_bwd(const __nv_bfloat16* __restrict__ W1, const __nv_bfloat16* __restrict__ W2, const float* __restrict__ dout,
                  const float* __restrict__ qpre, const float* __restrict__ u, float* __restrict__ dh, float* __restrict__ dW1,
                  double* __restrict__ dc1, double* __restrict__ dW2, double* __restrict__ dc2, int nlines, unsigned* status)
{
    constexpr int J = kW * kXK / kBT;  // pieces of 64 channels of a line per thread
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base;
    __shared__ __align__(16) float s_d[2][2][kG];  // dout of a line, rounded to BF16, double-buffered
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ch = (warp & 7) * 8 + (lane & 7);    // every piece of a thread has channel ch or ch + 64
    float q[2][J][8];
    float dv = 0.0f;                               // this thread's dout value (plane tid / 256, pixel tid % 256)
    float2* sums = reinterpret_cast<float2*>(sm + kQS) + tid;  // [kQSums], kBT apart: bs, g2 of channel ch; of ch + 64; dout
#pragma unroll
    for (int k = 0; k < kQSums; k++) sums[k * kBT] = make_float2(0.0f, 0.0f);
    auto load = [&](int line, int hf, int j) {
        const size_t o0 = (size_t)(line / kG) * kProj * kP + (size_t)(line % kG) * kG;
        int row, k8;
        x_piece<kBT>(tid, j, row, k8);
        ld8(q[hf][j], qpre + o0 + (size_t)(row + 64 * hf) * kP + k8 * 8);
    };
    auto load_d = [&](int line) {
        dv = __ldg(dout + ((size_t)(line / kG) * 2 + tid / kG) * kP + (size_t)(line % kG) * kG + tid % kG);
    };
    if (blockIdx.x < nlines) {
#pragma unroll
        for (int hf = 0; hf < 2; hf++)
#pragma unroll
            for (int j = 0; j < J; j++) load(blockIdx.x, hf, j);
        load_d(blockIdx.x);
    }
    tmem_alloc(&tmem_base, 256, warp);
    if (tid == 0) mbar_init(&bar);
    for (int i = tid; i < kProj * kW; i += kBT)  // W1 is [128][64]: element (o, c) to row c, K index o
        *reinterpret_cast<__nv_bfloat16*>(sm + kQW + kmajor_off(i % kW, i / kW, kProj / 8)) = W1[i];
    float w2[2][2];
#pragma unroll
    for (int hf = 0; hf < 2; hf++)
#pragma unroll
        for (int k = 0; k < 2; k++) w2[hf][k] = __bfloat162float(W2[k * kProj + ch + 64 * hf]);
    float acc[16];  // dW1 of channel (warp % 4) 32 + lane, 16 columns
#pragma unroll
    for (int k = 0; k < 16; k++) acc[k] = 0.0f;
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_base, base = smem_addr(sm);
    const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    uint32_t parity = 0;
    int held = 0, buf = 0;
    for (int line = blockIdx.x; line < nlines; line += gridDim.x) {
        const size_t o0 = (size_t)(line / kG) * kW * kP + (size_t)(line % kG) * kG;
        pair_add(sums[6 * kBT], dv);
        s_d[buf][tid / kG][tid % kG] = __bfloat162float(__float2bfloat16_rn(dv));
        if (line + (int)gridDim.x < nlines) load_d(line + gridDim.x);
#pragma unroll
        for (int j = 0; j < J; j++) {  // u: loaded here, its latency under the first channels' arithmetic
            int row, k8;
            x_piece<kBT>(tid, j, row, k8);
            float f[8];
            ld8(f, u + o0 + (size_t)row * kP + k8 * 8);
            *reinterpret_cast<uint4*>(sm + kQU + kmajor_off(row, k8 * 8, kXK)) = pack8(f);
        }
        __syncthreads();
        float bs[2] = {0.0f, 0.0f}, g2[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};  // of this line
#pragma unroll
        for (int j = 0; j < J; j++) {
            int row, k8;
            x_piece<kBT>(tid, j, row, k8);
            const float4 *p0 = reinterpret_cast<const float4*>(&s_d[buf][0][k8 * 8]), *p1 = reinterpret_cast<const float4*>(&s_d[buf][1][k8 * 8]);
            const float4 a0 = p0[0], a1 = p0[1], b0 = p1[0], b1 = p1[1];
            const float d0[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const float d1[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int hf = 0; hf < 2; hf++) {
                float f[8];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    float v, dg;
                    gelu_both(q[hf][j][k], v, dg);
                    f[k] = fmaf(w2[hf][1], d1[k], w2[hf][0] * d0[k]) * dg;
                    const float vb = __bfloat162float(__float2bfloat16_rn(v));
                    g2[hf][0] = fmaf(d0[k], vb, g2[hf][0]);
                    g2[hf][1] = fmaf(d1[k], vb, g2[hf][1]);
                }
                bs[hf] += sum8(f);
                if (line + (int)gridDim.x < nlines) load(line + gridDim.x, hf, j);  // the piece's registers are free
                const uint4 pk = pack8(f);
                const int o = row + 64 * hf;
                *reinterpret_cast<uint4*>(sm + kQA + kmajor_off(o, k8 * 8, kXK)) = pk;
                unsigned short* t = reinterpret_cast<unsigned short*>(sm + kQT + k8 * kQTs + (o >> 3) * 128 + (o & 7) * 2);
                const uint32_t w[4] = {pk.x, pk.y, pk.z, pk.w};
#pragma unroll
                for (int k = 0; k < 8; k++) t[k * 8] = (unsigned short)(w[k >> 1] >> (16 * (k & 1)));
            }
        }
#pragma unroll
        for (int hf = 0; hf < 2; hf++) {
            pair_add(sums[(3 * hf) * kBT], bs[hf]);
            pair_add(sums[(3 * hf + 1) * kBT], g2[hf][0]);
            pair_add(sums[(3 * hf + 2) * kBT], g2[hf][1]);
        }
        publish_smem();
        if (tid == 0) {
#pragma unroll
            for (int ks = 0; ks < kG / 16; ks++)  // dW1: K = 256 pixels
                mma_bf16(tmem + 128, smem_desc(base + kQA + ks * 256, 128, kXK * 128),
                         smem_desc(base + kQU + ks * 256, 128, kXK * 128), instr_desc(kW), ks > 0 || held > 0);
#pragma unroll
            for (int half = 0; half < 2; half++)
#pragma unroll
                for (int ks = 0; ks < kProj / 16; ks++)  // dh: K = 128 channels, 128 pixels each
                    mma_bf16(tmem + half * kW, smem_desc(base + kQT + half * (kM / 8) * kQTs + ks * 256, 128, kQTs),
                             smem_desc(base + kQW + ks * 256, 128, kProj / 8 * 128), instr_desc(kW), ks > 0);
            mma_commit(&bar);
        }
        if (!mma_wait(&bar, parity, status)) break;
        parity ^= 1;
        const bool flush = ++held == kFlush || line + (int)gridDim.x >= nlines;
        {
            // warp w: pixels 32 (w % 4) .. of half (w / 4) % 2, channels 32 (w / 8) ..
            const int half = (warp >> 2) & 1, c0 = (warp >> 3) * 32;
            float* o = dh + o0 + half * kM + (warp & 3) * 32 + lane;
#pragma unroll
            for (int c = 0; c < 32; c += 16) {
                float r[16];
                tmem_ld16(trow + half * kW + c0 + c, r);
#pragma unroll
                for (int k = 0; k < 16; k++) o[(size_t)(c0 + c + k) * kP] = r[k];
            }
        }
        if (flush) {
            float r[16];
            tmem_ld16(trow + 128 + (warp >> 2) * 16, r);
#pragma unroll
            for (int k = 0; k < 16; k++) acc[k] += r[k];
            held = 0;
        }
        buf ^= 1;
        retire_tile();
    }
    {
        float* o = dW1 + ((warp & 3) * 32 + lane) * kW + (warp >> 2) * 16;
#pragma unroll
        for (int k = 0; k < 16; k++) atomicAdd(o + k, acc[k]);
    }
#pragma unroll
    for (int k = 0; k < kQSums; k++) {
        double v = pair_value(sums[k * kBT]);
        if (k == 6)  // dout: a plane's 256 threads
            for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        const int o = ch + 64 * (k / 3);
        if (k == 6 ? lane == 0 : lane < 8)
            atomicAdd(k == 6 ? dc2 + tid / kG : k % 3 == 0 ? dc1 + o : dW2 + (k % 3 - 1) * kProj + o, v);
    }
    tmem_free(tmem, 256, warp);
}

// ---------------------------------------------------------------------------
// The projection head: q = gelu(W1 h + c1) (128 channels), out = W2 q + c2 (2
// channels).  The 2-channel product is two FMAs per value in the epilogue of
// the first, on q rounded to BF16 as the product rounds it, so inference
// neither stores q (537 MB per batch of 16) nor reads it back: 230 us for the
// first product and 381 us for a GEMM of N = 2 before.  keep: training stores
// the pre-activation, from which the backward pass forms q again.
// ---------------------------------------------------------------------------
constexpr uint32_t kPA = kProj * kW * 2, kPBytes = kPA + kM * kW * 2;

__global__ void __launch_bounds__(kThreads, 3)
    k_project(const __nv_bfloat16* __restrict__ W1, const float* __restrict__ c1, const __nv_bfloat16* __restrict__ W2,
              const float* __restrict__ c2, const float* __restrict__ X, float* __restrict__ qpre, float* __restrict__ out,
              int ntiles, unsigned* status, int keep)
{
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base;
    __shared__ float s_c1[kProj], s_w2[2][kProj], s_half[2][kM];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m = tid % kM, kc0 = tid / kM;
    float x[4][8];
    auto load_x = [&](int tile) {
        const float* src = X + (size_t)(tile / (int)(kP / kM)) * kW * kP + (size_t)(tile % (int)(kP / kM)) * kM + m;
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int q = 0; q < 8; q++) x[j][q] = __ldg(src + (size_t)((kc0 + 2 * j) * 8 + q) * kP);
    };
    if (blockIdx.x < ntiles) load_x(blockIdx.x);
    tmem_alloc(&tmem_base, 128, warp);
    if (tid == 0) mbar_init(&bar);
    for (int i = tid; i < kProj * kW; i += kThreads)
        *reinterpret_cast<__nv_bfloat16*>(sm + kmajor_off(i / kW, i % kW, kFK)) = W1[i];
    if (tid < kProj) {
        s_c1[tid] = c1[tid];
        s_w2[0][tid] = __bfloat162float(W2[tid]);
        s_w2[1][tid] = __bfloat162float(W2[kProj + tid]);
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_base, base = smem_addr(sm);
    const float o0 = c2[0], o1 = c2[1];
    uint32_t parity = 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
#pragma unroll
        for (int j = 0; j < 4; j++)
            *reinterpret_cast<uint4*>(sm + kPA + kmajor_off(m, (kc0 + 2 * j) * 8, kFK)) = pack8(x[j]);
        publish_smem();
        if (tile + (int)gridDim.x < ntiles) load_x(tile + gridDim.x);
        if (tid == 0) {
#pragma unroll
            for (int ks = 0; ks < kW / 16; ks++)
                mma_bf16(tmem, smem_desc(base + kPA + ks * 256, 128, kFK * 128),
                         smem_desc(base + ks * 256, 128, kFK * 128), instr_desc(kProj), ks > 0);
            mma_commit(&bar);
        }
        if (!mma_wait(&bar, parity, status)) break;
        parity ^= 1;
        const int g = warp & 3, ch = warp >> 2;
        const uint32_t trow = tmem + ((uint32_t)(g * 32) << 16);
        const size_t b = tile / (int)(kP / kM), p = (size_t)(tile % (int)(kP / kM)) * kM + g * 32 + lane;
        float y0 = 0.0f, y1 = 0.0f;
#pragma unroll 1
        for (int c0 = ch * (kProj / 2); c0 < (ch + 1) * (kProj / 2); c0 += 16) {
            float r[16];
            tmem_ld16(trow + c0, r);
#pragma unroll
            for (int q = 0; q < 16; q++) {
                const float u = r[q] + s_c1[c0 + q], v = gelu_f(u);
                if (keep) qpre[(b * kProj + c0 + q) * kP + p] = u;
                const float vb = __bfloat162float(__float2bfloat16_rn(v));
                y0 = fmaf(s_w2[0][c0 + q], vb, y0);
                y1 = fmaf(s_w2[1][c0 + q], vb, y1);
            }
        }
        if (ch == 1) {
            s_half[0][g * 32 + lane] = y0;
            s_half[1][g * 32 + lane] = y1;
        }
        retire_tile();  // (also orders the upper half's sums)
        if (ch == 0) {
            out[(b * 2) * kP + p] = (y0 + s_half[0][g * 32 + lane]) + o0;
            out[(b * 2 + 1) * kP + p] = (y1 + s_half[1][g * 32 + lane]) + o1;
        }
    }
    tmem_free(tmem, 128, warp);
}

template <typename K>
cudaError_t allow_smem(K k, uint32_t bytes)
{
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

int sm_count()
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 1;
    return sms;
}

}  // namespace umma

// The shape the fused forward kernels are compiled for.
bool fused_supported(int grid, int modes, int width, int proj, int nout)
{
    return grid == umma::kG && modes == umma::kModes && width == umma::kW && proj == umma::kProj && nout == 2;
}

cudaError_t xdft_fused(const __nv_bfloat16* F, const float* H, float* a, int B, unsigned* status, cudaStream_t st)
{
    using namespace umma;
    const cudaError_t e = allow_smem(k_xdft, 2 * kXBytes);
    if (e != cudaSuccess) return e;
    const int lines = B * kG, grid = lines < 2 * sm_count() ? lines : 2 * sm_count();
    k_xdft<<<grid, kThreads, 2 * kXBytes, st>>>(F, H, a, lines, (long)B * kW * kModes, status);
    return cudaGetLastError();
}

// z = F a, F 64 x 512 (FyAB); split: K in four runs of 128 (dy)
cudaError_t yfwd_fused(const __nv_bfloat16* F, const float* a, float* z, int B, unsigned* status, bool split, cudaStream_t st)
{
    using namespace umma;
    const auto kern = split ? k_yfwd<true> : k_yfwd<false>;
    const cudaError_t e = allow_smem(kern, kYBytes);
    if (e != cudaSuccess) return e;
    const long P = (long)B * kW * kModes;
    const int tiles = (int)(P / kM), grid = tiles < 2 * sm_count() ? tiles : 2 * sm_count();
    kern<<<grid, kThreads, kYBytes, st>>>(F, a, z, P, tiles, status);
    return cudaGetLastError();
}

// bb = G y, G 512 x 64 (GyBig)
cudaError_t yinv_fused(const __nv_bfloat16* G, const float* y, float* bb, int B, unsigned* status, cudaStream_t st)
{
    using namespace umma;
    const cudaError_t e = allow_smem(k_yinv, kIBytes);
    if (e != cudaSuccess) return e;
    const long P = (long)B * kW * kModes;
    const int tiles = (int)(P / kM), grid = 4 * (tiles < sm_count() ? tiles : sm_count());
    k_yinv<<<grid, kThreads, kIBytes, st>>>(G, y, bb, P, tiles, status);
    return cudaGetLastError();
}

namespace umma {
template <bool TW, bool SPEC, int KX, bool DFT>
cudaError_t launch_fourier(const __nv_bfloat16* W, const __nv_bfloat16* Gt, const float* X, const float* bb, float* U, float* act,
                           const float* bias, const __nv_bfloat16* F, float* a, int B, unsigned* status, bool write_u,
                           cudaStream_t st)
{
    constexpr uint32_t bytes = FourierSmem<SPEC, KX, DFT>::bytes;
    const auto kern = k_fourier<TW, SPEC, KX, DFT>;
    const cudaError_t e = allow_smem(kern, bytes);
    if (e != cudaSuccess) return e;
    const int lines = B * kG, ctas = (SPEC ? 2 : 3) * sm_count(), grid = lines < ctas ? lines : ctas;
    kern<<<grid, kThreads, bytes, st>>>(W, Gt, X, bb, U, act, bias, F, a, lines, (long)B * kW * kModes, status, write_u);
    return cudaGetLastError();
}
}  // namespace umma

// h = W x + bias of 8 input planes, and its forward DFT along x (F: 2 m x G).
bool lift_supported(int nin) { return nin == 8; }

cudaError_t lift_fused(const __nv_bfloat16* W, const float* X, float* h, const float* bias, const __nv_bfloat16* F, float* a,
                       int B, unsigned* status, cudaStream_t st)
{
    return umma::launch_fourier<false, false, 8, true>(W, nullptr, X, nullptr, h, nullptr, bias, F, a, B, status, true, st);
}

// act NULL: the last layer (no activation, and no layer that wants its DFT).
cudaError_t fourier_fused(const __nv_bfloat16* W, const __nv_bfloat16* Gt, const float* X, const float* bb, float* U,
                          float* act, const float* bias, const __nv_bfloat16* F, float* a, int B, unsigned* status,
                          bool write_u, cudaStream_t st)
{
    if (!act)
        return umma::launch_fourier<false, true, umma::kW, false>(W, Gt, X, bb, U, act, bias, nullptr, nullptr, B, status, true,
                                                                  st);
    return umma::launch_fourier<false, true, umma::kW, true>(W, Gt, X, bb, U, act, bias, F, a, B, status, write_u, st);
}

// dX = W^T dU + the transposed forward DFT along x of da (Fx: G x 2 m)
cudaError_t fourier_bwd_fused(const __nv_bfloat16* W, const __nv_bfloat16* Fx, const float* dU, const float* da, float* dX,
                              int B, unsigned* status, cudaStream_t st)
{
    return umma::launch_fourier<true, true, umma::kW, false>(W, Fx, dU, da, dX, nullptr, nullptr, nullptr, nullptr, B, status,
                                                             true, st);
}

// u NULL: no activation (du is dh and is not written).  dW and db accumulate;
// db, and dc1, dW2 and dc2 below, are FP64 sums that the caller clears.
cudaError_t layer_bwd_fused(const __nv_bfloat16* Gx, const float* dh, const float* u, const float* h, float* du, float* dbb,
                            float* dW, double* db, int B, unsigned* status, cudaStream_t st)
{
    using namespace umma;
    const int lines = B * kG, grid = lines < sm_count() ? lines : sm_count();
    const long Nc = (long)B * kW * kModes;
    auto go = [&](auto kern) {
        const cudaError_t e = allow_smem(kern, kLBytes);
        if (e != cudaSuccess) return e;
        kern<<<grid, kBT, kLBytes, st>>>(Gx, dh, u, h, du, dbb, dW, db, lines, Nc, status);
        return cudaGetLastError();
    };
    return u ? go(k_layer_bwd<true, true, kW>) : go(k_layer_bwd<false, true, kW>);
}

// The lift's gradients: dW (64 x nin) += dh x^T, db += sum dh.
bool lift_bwd_supported(int nin) { return nin == 8; }

cudaError_t lift_bwd_fused(const float* dh, const float* x, float* dW, double* db, int B, unsigned* status, cudaStream_t st)
{
    using namespace umma;
    const cudaError_t e = allow_smem(k_layer_bwd<false, false, 8>, kLBytes);
    if (e != cudaSuccess) return e;
    const int lines = B * kG, grid = lines < sm_count() ? lines : sm_count();
    k_layer_bwd<false, false, 8><<<grid, kBT, kLBytes, st>>>(nullptr, dh, nullptr, x, nullptr, nullptr, dW, db, lines,
                                                             (long)B * kW * kModes, status);
    return cudaGetLastError();
}

cudaError_t project_bwd_fused(const __nv_bfloat16* W1, const __nv_bfloat16* W2, const float* dout, const float* qpre,
                              const float* u, float* dh, float* dW1, double* dc1, double* dW2, double* dc2, int B,
                              unsigned* status, cudaStream_t st)
{
    using namespace umma;
    const cudaError_t e = allow_smem(k_project_bwd, kQBytes);
    if (e != cudaSuccess) return e;
    const int lines = B * kG, grid = lines < sm_count() ? lines : sm_count();
    k_project_bwd<<<grid, kBT, kQBytes, st>>>(W1, W2, dout, qpre, u, dh, dW1, dc1, dW2, dc2, lines, status);
    return cudaGetLastError();
}

cudaError_t project_fused(const __nv_bfloat16* W1, const float* c1, const __nv_bfloat16* W2, const float* c2,
                          const float* X, float* qpre, float* out, int B, unsigned* status, bool keep,
                          cudaStream_t st)
{
    using namespace umma;
    const cudaError_t e = allow_smem(k_project, kPBytes);
    if (e != cudaSuccess) return e;
    const int tiles = (int)(B * (kP / kM)), grid = tiles < 3 * sm_count() ? tiles : 3 * sm_count();
    k_project<<<grid, kThreads, kPBytes, st>>>(W1, c1, W2, c2, X, qpre, out, tiles, status, keep);
    return cudaGetLastError();
}

}  // namespace atmwfs
