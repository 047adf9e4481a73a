// Learned initialiser: a small 3-D convolutional encoder with an MLP head that reads a
// fixed/moving pair downsampled to 32³ and proposes the 12 affine parameters a
// registration starts from. It is trained on pairs the library generates and
// registers itself (labels: the regular-step optimizer's converged result).
//
//   input 2 × 32³ → conv 3³ stride 2 (+ReLU): 16 × 16³ → 32 × 8³ → 64 × 4³ → 128 × 2³
//   → flatten 1024 → fc 256 (+ReLU) → fc 12
//
// Every convolution runs as a GEMM over im2col rows (channels-last activations; the
// column index of an im2col row is ((kz·3 + ky)·3 + kx)·Cin + c), forward and
// backward, on the tcgen05 BF16 GEMM (gemm_tma.cuh) with FP32 accumulation: forward
// Y = Xcol·Wᵀ; weight gradient dW = dYᵀ·Xcol; input gradient dXcol = dY·W, gathered
// back to the input grid (col2im as a gather, so deterministic). Master weights, biases
// and Adam moments are FP32. The 31 launches of a step are programmatic dependents of one
// another, so that each one's launch and set-up overlap the end of the one before: with
// the stores by TMA a step takes 274 µs for 64 pairs and 140 µs for one (about 390 µs for 64
// before both). No reference counterpart.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "gemm_tc.cuh"
#include "gemm_tma.cuh"
#include "internal.h"
#include "pdl.cuh"

namespace mi {

namespace {

template <int NT>
cudaError_t launch_gemm(int M, int N, int K, const __nv_bfloat16* A, int lda, const __nv_bfloat16* B, int ldb, float* C,
                        int ldc, int splits, unsigned int* err, cudaStream_t st) {
    const size_t sm = tc::gemm_smem<NT>();
    cudaError_t e = cudaFuncSetAttribute(tc::k_gemm_tn<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    dim3 grid((M + tc::TILE_M - 1) / tc::TILE_M, (N + NT - 1) / NT, splits);
    tc::k_gemm_tn<NT><<<grid, tc::THREADS, sm, st>>>(M, N, K, A, lda, B, ldb, C, ldc, err);
    return cudaGetLastError();
}

int n_tile(int N) { return N <= 16 ? 16 : N <= 32 ? 32 : N <= 64 ? 64 : 128; }

// One operand of a product: element (r, k) at r·ld + k, or with k_rows at k·ld + r.
struct Operand {
    const __nv_bfloat16* p;
    int ld;
    bool k_rows;
};

// The operand's tiles, `box` rows × 64 k (64 × 64 with k_rows), 128-byte swizzle; k and rows
// past the ends read as zero. False where TMA cannot read it (pitch or base not a
// multiple of 16 bytes).
bool operand_map(CUtensorMap* map, const Operand& o, int rows, int K, int box) {
    if (o.ld % 8 != 0 || ((uintptr_t)o.p & 15) != 0 || !tensor_map_encoder()) return false;
    const cuuint64_t dim[2] = {(cuuint64_t)(o.k_rows ? rows : K), (cuuint64_t)(o.k_rows ? K : rows)};
    const cuuint64_t stride[1] = {(cuuint64_t)o.ld * 2};
    const cuuint32_t bx[2] = {64, (cuuint32_t)(o.k_rows ? 64 : box)}, es[2] = {1, 1};
    static_assert(tc::TILE_K == 64, "tiles of 64 k");
    return tensor_map_encoder()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(o.p), dim, stride, bx,
                                es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The map of a product's output (rows × N, `splits` of them one after another) in blocks of 32
// rows × min(nt, 32) columns, swizzled by their rows' bytes. False where TMA cannot
// write it.
bool output_map(CUtensorMap* map, const tc::Epilogue& E, int M, int N, int splits, int nt) {
    const bool f32 = E.C != nullptr;
    const cuuint64_t size = f32 ? 4 : 2, pitch = (cuuint64_t)(f32 ? E.ldc : E.ldx) * size;
    void* p = f32 ? (void*)E.C : (void*)E.X;
    // a row that ended inside 16 bytes would clear the rest of them
    if (pitch % 16 != 0 || (cuuint64_t)N * size % 16 != 0 || ((uintptr_t)p & 15) != 0 || !tensor_map_encoder()) return false;
    const cuuint32_t w = (cuuint32_t)std::min(nt, 32), row = w * (cuuint32_t)size;
    const cuuint64_t dim[3] = {(cuuint64_t)N, (cuuint64_t)M, (cuuint64_t)splits}, stride[2] = {pitch, pitch * (cuuint64_t)M};
    const cuuint32_t bx[3] = {w, 32, 1}, es[3] = {1, 1, 1};
    return tensor_map_encoder()(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, p, dim,
                                stride, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                row == 128  ? CU_TENSOR_MAP_SWIZZLE_128B
                                : row == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                            : CU_TENSOR_MAP_SWIZZLE_32B,
                                CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int NT, bool AK, bool BK, int MT = 1>
cudaError_t launch_tma(mi_context* ctx, int M, int N, int K, const CUtensorMap& a, const CUtensorMap& b,
                       const CUtensorMap& out, const tc::Epilogue& E, int splits, unsigned int* err) {
    constexpr uint32_t sm = tc::TmaShape<NT, MT>::SMEM;
    if (raise_smem_limit(ctx, (const void*)tc::k_gemm_tma<NT, AK, BK, MT>, sm) != MI_OK) return cudaErrorInvalidValue;
    const int64_t items = (int64_t)((M + MT * tc::TILE_M - 1) / (MT * tc::TILE_M)) * ((N + NT - 1) / NT) * splits;
    const int grid = (int)std::min<int64_t>(items, ctx->num_sms);
    return pdl::launch(tc::k_gemm_tma<NT, AK, BK, MT>, grid, tc::TMA_THREADS, sm, ctx->stream, a, b, out, M, N, K, E, splits, err);
}

// The N tile of the TMA kernel. Its tiles are 128 × 256 where that leaves at least as few
// columns of padding and as full a last round of CTAs as 128 × 128, which needs half
// as much again of shared-memory bandwidth per product.
int tma_n_tile(mi_context* ctx, int M, int N, int splits) {
    if (N <= 128) return n_tile(N);
    const int64_t mt = (M + tc::TILE_M - 1) / tc::TILE_M;
    auto rounds = [&](int nt) {
        const int64_t items = mt * ((N + nt - 1) / nt) * splits;
        return (items + ctx->num_sms - 1) / ctx->num_sms;
    };
    return 2 * rounds(256) * 3 <= rounds(128) * 4 ? 256 : 128;
}

// Whether tiles of 256 × 256 (two blocks of 128 rows on one B tile) take a product of
// 256-column tiles. They bring 64 KB a k tile from L2 for twice the work of 48 KB, but their
// accumulators fill the tensor memory, so a tile's stores (about eight k tiles' time) do not
// overlap the next one's products. Two blocks against one: 4096³ 109 against 118 µs, 8192³
// 717 against 825, 3000³ 58 against 75, 4096 × 2304 × 2056 48 against 59, 1300 × 4100 × 1032
// 35 against 41; 4096 × 4096 × 1024, where the rule's sides are equal, 48.7 against 48.2.
bool two_blocks(mi_context* ctx, int M, int N, int K, int splits) {
    const int64_t nt = (N + 255) / 256, kt = ((K + tc::TILE_K - 1) / tc::TILE_K + splits - 1) / splits;
    auto rounds = [&](int rows) {
        const int64_t items = (M + rows - 1) / rows * nt * splits;
        return (items + ctx->num_sms - 1) / ctx->num_sms;
    };
    return rounds(256) * 64 * (kt + 8) < rounds(128) * 48 * kt;
}

// The product by TMA: E's outputs, or with splits > 1 the K slices' partial products one
// after another in E.C (M × ldc each). cudaErrorNotSupported where TMA cannot read an
// operand. Both operands may be k_rows, or B alone.
cudaError_t product(mi_context* ctx, int M, int N, int K, const Operand& A, const Operand& B, tc::Epilogue E,
                    int splits, unsigned int* err) {
    int nt = tma_n_tile(ctx, M, N, splits);
    if (B.k_rows) nt = std::max(nt, 64);
    CUtensorMap a, b, out = {};
    if (!operand_map(&a, A, M, K, tc::TILE_M) || !operand_map(&b, B, N, K, nt)) return cudaErrorNotSupported;
    E.tma = output_map(&out, E, M, N, splits, nt);
    if (!E.tma && !E.C) return cudaErrorNotSupported;
#define MI_PRODUCT(NT, AK, BK) return launch_tma<NT, AK, BK>(ctx, M, N, K, a, b, out, E, splits, err)
    if (A.k_rows) {
        switch (nt) {
            case 64: MI_PRODUCT(64, true, true);
            case 128: MI_PRODUCT(128, true, true);
            default: MI_PRODUCT(256, true, true);
        }
    }
    if (B.k_rows) {
        switch (nt) {
            case 64: MI_PRODUCT(64, false, true);
            case 128: MI_PRODUCT(128, false, true);
            default: MI_PRODUCT(256, false, true);
        }
    }
    switch (nt) {
        case 16: MI_PRODUCT(16, false, false);
        case 32: MI_PRODUCT(32, false, false);
        case 64: MI_PRODUCT(64, false, false);
        case 128: MI_PRODUCT(128, false, false);
        default:
            if (two_blocks(ctx, M, N, K, splits))
                return launch_tma<256, false, false, 2>(ctx, M, N, K, a, b, out, E, splits, err);
            MI_PRODUCT(256, false, false);
    }
#undef MI_PRODUCT
}

// C = A·Bᵀ for operands of any pitch: those TMA cannot read take k_gemm_tn's plain loads.
// Same slices, same order of accumulation, same bits.
cudaError_t gemm_dispatch(mi_context* ctx, int M, int N, int K, const __nv_bfloat16* A, int lda, const __nv_bfloat16* B,
                          int ldb, float* C, int ldc, int splits, unsigned int* err) {
    const cudaError_t e = product(ctx, M, N, K, Operand{A, lda, false}, Operand{B, ldb, false},
                                  tc::Epilogue{C, ldc, nullptr, nullptr, 0, 0, 0}, splits, err);
    if (e != cudaErrorNotSupported) return e;
    cudaStream_t st = ctx->stream;
    switch (n_tile(N)) {
        case 16: return launch_gemm<16>(M, N, K, A, lda, B, ldb, C, ldc, splits, err, st);
        case 32: return launch_gemm<32>(M, N, K, A, lda, B, ldb, C, ldc, splits, err, st);
        case 64: return launch_gemm<64>(M, N, K, A, lda, B, ldb, C, ldc, splits, err, st);
        default: return launch_gemm<128>(M, N, K, A, lda, B, ldb, C, ldc, splits, err, st);
    }
}

constexpr int NCONV = 4;
constexpr int CH[NCONV + 1] = {2, 16, 32, 64, 128};
constexpr int DIM[NCONV + 1] = {32, 16, 8, 4, 2};
constexpr int FC1_IN = 128 * 8, FC1_OUT = 256, FC2_OUT = 12;
constexpr int NLAYER = NCONV + 2;

inline int kraw(int l) { return 27 * CH[l]; }          // im2col width of conv l (0-based)
// padded to 16-byte rows, the first layer's to a whole tile: its 262,144 rows' product (64
// pairs) takes 18.5–20.3 µs where TMA fills 56 columns up to 64, 12.7 µs with 64 stored (the
// others' last tiles are one in seven or fewer)
inline int kpad(int l) { return l == 0 ? 64 : (kraw(l) + 7) & ~7; }

inline int grid1(int64_t n) {
    const int64_t g = (n + 255) / 256;
    return (int)(g < 65535 * 16 ? (g < 1 ? 1 : g) : 65535 * 16);
}

#define GSTRIDE(i, n) for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

__global__ void k_to_bf16(const float* __restrict__ in, __nv_bfloat16* __restrict__ out, int64_t n) {
    GSTRIDE(i, n) out[i] = __float2bfloat16(in[i]);
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// im2col of a channels-last volume (B × D³ × CIN) for a 3³ stride-2 pad-1 convolution: row
// (b, z, y, x) of the D/2 output grid, column ((kz·3+ky)·3+kx)·CIN + c, zeros to KP columns.
// A thread fills eight columns (16 bytes): eight channels of one tap, or, in the first
// layer, both channels of four taps, read from the FP32 input and rounded here. Bound by
// the bytes written (34 and 28 MB in the two large layers for 64 pairs: 17 and 10.5 µs with
// cold caches; 22.6 and 13.2 µs with 64-bit indices over all pairs). A CTA's rows are the
// same in every pair, blockIdx.y. The caller's input may start on any float: a voxel's two
// channels are one load only where it starts on eight bytes.
template <int D, int CIN, int KP, typename T>
__global__ void __launch_bounds__(256) k_im2col(const T* x, int B, __nv_bfloat16* col) {
    constexpr uint32_t Do = D / 2, PARTS = KP / 8, N = Do * Do * Do * PARTS;
    pdl::launch_dependents();
    const uint32_t i = blockIdx.x * 256 + threadIdx.x;  // of a sample's rows
    pdl::wait_previous();
    if (i >= N) return;
    const uint32_t part = i % PARTS, row = i / PARTS;
    const int xo = (int)(row % Do), yo = (int)(row / Do % Do), zo = (int)(row / (Do * Do));
    int off[CIN == 2 ? 4 : 1];  // the input voxel under the tap, -1: none
#pragma unroll
    for (int q = 0; q < (CIN == 2 ? 4 : 1); ++q) {
        const int t = CIN == 2 ? (int)part * 4 + q : (int)(part / (CIN / 8));
        const int xi = 2 * xo + t % 3 - 1, yi = 2 * yo + t / 3 % 3 - 1, zi = 2 * zo + t / 9 - 1;
        off[q] = t < 27 && (unsigned)xi < (unsigned)D && (unsigned)yi < (unsigned)D && (unsigned)zi < (unsigned)D
                     ? (zi * D + yi) * D + xi
                     : -1;
    }
    const bool paired = CIN != 2 || (reinterpret_cast<uintptr_t>(x) & 7) == 0;
    for (int b = blockIdx.y; b < B; b += gridDim.y) {
        const T* in = x + (size_t)b * (D * D * D * CIN);
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if constexpr (CIN == 2) {
            uint32_t w[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float2 f = make_float2(0.f, 0.f);
                if (off[q] >= 0) {
                    const T* at = in + 2 * off[q];
                    f = paired ? __ldca(reinterpret_cast<const float2*>(at)) : make_float2(__ldca(at), __ldca(at + 1));
                }
                w[q] = pack_bf16(f.x, f.y);
            }
            v = make_uint4(w[0], w[1], w[2], w[3]);
        } else {
            if (off[0] >= 0) v = __ldca(reinterpret_cast<const uint4*>(in + (size_t)off[0] * CIN + part % (CIN / 8) * 8));
        }
        reinterpret_cast<uint4*>(col)[(size_t)b * N + i] = v;
    }
}

// The end of a layer's forward product that was split over K: the slices summed in order,
// the bias, ReLU, BF16.
__global__ void k_slices_act(const float* part, int splits, int64_t mn, const float* bias, int cols, __nv_bfloat16* x) {
    pdl::launch_dependents();
    pdl::wait_previous();
    GSTRIDE(i, mn) {
        float acc = 0.0f;
        for (int s = 0; s < splits; ++s) acc += __ldcg(part + (int64_t)s * mn + i);
        x[i] = __float2bfloat16(tc::relu(acc + __ldca(bias + i % cols)));
    }
}

// The gradient dZ of the layer below from that of a layer's input: dx through the ReLU (its
// output a has no sign where its input was positive: tc::relu), as BF16 for the next products, and the
// CTA's column sums (the bias gradient) of the FP32 values into part[CTA]. dx comes
// from the layer's product dcol: for a fully connected layer it is dcol itself (D = 0); for
// a convolution over D³ inputs of C channels it is the transpose of im2col as a gather,
// the output voxels and taps that read the input voxel, in a fixed order. A thread keeps
// four channels, so that its sums stay in registers, and requests all of a voxel's up to
// eight values before it adds them: 57 MB of the first layer's dcol in 30 µs with cold
// caches, 43 µs tap by tap. (Gather, ReLU, conversion and sums were five launches; the
// sums, 4,096 rows a thread in order, took 0.9–1.1 ms each.)
template <int D, int C, int KP>
__global__ void __launch_bounds__(256) k_back_act(const float* dcol, const __nv_bfloat16* a, int64_t rows,
                                                  __nv_bfloat16* dzb, float* part) {
    constexpr int G = C / 4;  // threads a row
    static_assert(256 % G == 0, "a thread's channels stay the same");
    __shared__ float4 sums[256];
    pdl::launch_dependents();
    pdl::wait_previous();
    const int c = (threadIdx.x % G) * 4;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int64_t r = ((int64_t)blockIdx.x * 256 + threadIdx.x) / G; r < rows; r += (int64_t)gridDim.x * (256 / G)) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if constexpr (D == 0) {
            v = __ldcg(reinterpret_cast<const float4*>(dcol + r * C + c));
        } else {
            constexpr int Do = D / 2;
            const uint32_t in = (uint32_t)(r % (D * D * D));
            const int xi = (int)(in % D), yi = (int)(in / D % D), zi = (int)(in / (D * D));
            const int64_t b = r / (D * D * D);
            // Per axis an even input voxel is read by tap 1 of output i/2 alone, an odd one by tap
            // 0 of the output after it (if there is one) and by tap 2 of the one before: two
            // slots an axis, eight loads at once.
            int o[3][2], tap[3][2];
            const int at[3] = {zi, yi, xi};
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const int odd = at[d] & 1;
                o[d][0] = (at[d] + odd) >> 1;
                tap[d][0] = odd ? 0 : 1;
                if (o[d][0] >= Do) tap[d][0] = -1;
                o[d][1] = at[d] >> 1;
                tap[d][1] = odd ? 2 : -1;
            }
            float4 t[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int z = q >> 2, y = (q >> 1) & 1, xx = q & 1;
                t[q] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (tap[0][z] >= 0 && tap[1][y] >= 0 && tap[2][xx] >= 0) {
                    const int64_t row = ((b * Do + o[0][z]) * Do + o[1][y]) * Do + o[2][xx];
                    t[q] = __ldcg(reinterpret_cast<const float4*>(dcol + row * KP +
                                                                  ((tap[0][z] * 3 + tap[1][y]) * 3 + tap[2][xx]) * C + c));
                }
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) v = make_float4(v.x + t[q].x, v.y + t[q].y, v.z + t[q].z, v.w + t[q].w);
        }
        const uint2 act = __ldcg(reinterpret_cast<const uint2*>(a + r * C + c));
        v.x = act.x & 0x8000u ? 0.f : v.x;
        v.y = act.x & 0x80000000u ? 0.f : v.y;
        v.z = act.y & 0x8000u ? 0.f : v.z;
        v.w = act.y & 0x80000000u ? 0.f : v.w;
        *reinterpret_cast<uint2*>(dzb + r * C + c) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
        sum = make_float4(sum.x + v.x, sum.y + v.y, sum.z + v.z, sum.w + v.w);
    }
    sums[threadIdx.x] = sum;
    __syncthreads();
    if (threadIdx.x < G) {
        for (int t = threadIdx.x + G; t < 256; t += G) {
            const float4 o = sums[t];
            sum = make_float4(sum.x + o.x, sum.y + o.y, sum.z + o.z, sum.w + o.w);
        }
        *reinterpret_cast<float4*>(part + (int64_t)blockIdx.x * C + c) = sum;
    }
}

// loss = mean (out − t)², dout = 2(out − t)/n as BF16 rows of ld, its column sums into
// colsum (one CTA, fixed order)
__global__ void __launch_bounds__(256) k_mse(const float* out, const float* t, int rows, int cols, __nv_bfloat16* dzb, int ld,
                                             float* colsum, float* loss) {
    __shared__ float red[256];
    pdl::launch_dependents();
    pdl::wait_previous();
    const int n = rows * cols;
    float acc = 0.0f;
    for (int i = threadIdx.x; i < n; i += 256) {
        const float d = __ldca(out + i) - __ldca(t + i);
        dzb[i / cols * ld + i % cols] = __float2bfloat16(2.0f * d / (float)n);
        acc += d * d;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) *loss = red[0] / (float)n;
    __syncthreads();
    // sixteen threads a column, their sums in order
    for (int c0 = 0; c0 < cols; c0 += 16) {
        const int c = c0 + threadIdx.x / 16, q = threadIdx.x % 16;
        float s = 0.0f;
        if (c < cols)
            for (int r = q; r < rows; r += 16) s += 2.0f * (__ldca(out + r * cols + c) - __ldca(t + r * cols + c)) / (float)n;
        red[threadIdx.x] = s;
        __syncthreads();
        if (q == 0 && c < cols) {
            for (int k = 1; k < 16; ++k) s += red[threadIdx.x + k];
            colsum[c] = s;
        }
        __syncthreads();
    }
}

// One tensor of parameters at the end of a training step.
struct Tensor {
    float *w, *g, *m, *v;
    __nv_bfloat16* wb;   // its BF16 copy (weights)
    const float* part;   // partial gradients to sum, n apart (null: g holds the gradient)
    int n, parts;
    int block0;          // its first CTA
};
struct Tensors {
    Tensor t[12];
};
// Tensors with at least this many partials take eight warps to each element.
constexpr int WIDE_PARTS = 24;
inline int tensor_blocks(int n, int parts) { return parts >= WIDE_PARTS ? (n + 31) / 32 : (n + 255) / 256; }

// The gradients' partials summed in a fixed order, then (lr > 0) Adam on the FP32 master
// values and their BF16 copies: one launch for all layers (it was a sum per split
// product, twelve Adam launches and twelve conversions and transposes).
__global__ void __launch_bounds__(256) k_update(const __grid_constant__ Tensors T, float lr, float b1, float b2, float c1,
                                                float c2, float eps) {
    __shared__ float red[8][32];
    int k = 0;
    while (k < 11 && (int)blockIdx.x >= T.t[k + 1].block0) ++k;
    const Tensor& t = T.t[k];
    const int blk = (int)blockIdx.x - t.block0;
    int i;
    float g = 0.0f;
    pdl::launch_dependents();
    pdl::wait_previous();
    if (t.parts >= WIDE_PARTS) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        i = blk * 32 + lane;
        if (i < t.n)
#pragma unroll 8
            for (int s = warp; s < t.parts; s += 8) g += __ldcg(t.part + (int64_t)s * t.n + i);
        red[warp][lane] = g;
        __syncthreads();
        if (warp > 0) return;
        for (int q = 1; q < 8; ++q) g += red[q][lane];
        if (i >= t.n) return;
    } else {
        i = blk * 256 + threadIdx.x;
        if (i >= t.n) return;
        if (t.part)
#pragma unroll 4
            for (int s = 0; s < t.parts; ++s) g += __ldcg(t.part + (int64_t)s * t.n + i);
        else
            g = t.g[i];
    }
    if (t.part) t.g[i] = g;
    if (!(lr > 0.0f)) return;
    const float mi = b1 * t.m[i] + (1.0f - b1) * g;
    const float vi = b2 * t.v[i] + (1.0f - b2) * g * g;
    t.m[i] = mi;
    t.v[i] = vi;
    const float w = t.w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    t.w[i] = w;
    if (t.wb) t.wb[i] = __float2bfloat16(w);
}

// out[i] = Σ_s part[s·mn + i], slices in order
__global__ void k_sum_slices(const float* __restrict__ part, int splits, int64_t mn, float* __restrict__ out) {
    GSTRIDE(i, mn) {
        float acc = 0.0f;
        for (int s = 0; s < splits; ++s) acc += part[(int64_t)s * mn + i];
        out[i] = acc;
    }
}

// K slices for a GEMM whose M × N tiles alone would leave most SMs idle: about two
// CTAs per SM in all, at least 4 k tiles per slice
int k_splits(int M, int N, int K) {
    const int tiles = ((M + tc::TILE_M - 1) / tc::TILE_M) * ((N + n_tile(N) - 1) / n_tile(N));
    const int ktiles = (K + tc::TILE_K - 1) / tc::TILE_K;
    int s = (296 + tiles - 1) / tiles;
    s = std::min(s, std::max(1, ktiles / 4));
    return std::max(1, s);
}

// mean and standard deviation of an n-voxel image (one CTA, FP64), then the image
// normalised into channel `ch` of a channels-last two-channel volume
__global__ void k_normalise(const float* __restrict__ img, int64_t n, float* __restrict__ out, int ch) {
    __shared__ double s1[256], s2[256];
    double a = 0.0, b = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const double v = img[i];
        a += v;
        b += v * v;
    }
    s1[threadIdx.x] = a;
    s2[threadIdx.x] = b;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            s1[threadIdx.x] += s1[threadIdx.x + s];
            s2[threadIdx.x] += s2[threadIdx.x + s];
        }
        __syncthreads();
    }
    const double mean = s1[0] / (double)n;
    const double var = fmax(s2[0] / (double)n - mean * mean, 1e-12);
    const float inv = (float)(1.0 / sqrt(var));
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) out[2 * i + ch] = (float)((img[i] - mean)) * inv;
}

struct Layer {
    int out, in, kp;      // W is out × kp (FP32 master; columns ≥ the true width stay 0)
    float *w, *b, *gw, *gb, *mw, *vw, *mb, *vb;
    __nv_bfloat16* wb;    // BF16 W
    __nv_bfloat16* dzb;   // dZ (rows × dz_ld(out)) of the last training step
    float* wpart;         // the K slices of its weight gradient (null: one slice)
    float* bpart;         // the CTAs' column sums of dZ
    int wparts, bparts;   // how many of either
};

// Row pitch of dZ: TMA wants multiples of 16 bytes.
inline int dz_ld(int out) { return (out + 7) & ~7; }

}  // namespace
}  // namespace mi

struct mi_initnet {
    mi::Held ctx;
    int max_batch = 0;
    mi::Layer L[mi::NLAYER] = {};
    int step = 0;
    // activations (sized for max_batch)
    __nv_bfloat16* col[mi::NCONV] = {};        // im2col rows
    __nv_bfloat16* xb[mi::NLAYER] = {};        // activations (BF16): conv outputs, fc1
    float* out = nullptr;                      // fc2 output
    float* dcol = nullptr;                     // a layer's input gradient, in im2col columns
    float* slices = nullptr;                   // split-K partial products of a forward layer
    // pinned host words and their device addresses: [0] raised by a GEMM whose wait gave up,
    // [1] the loss
    unsigned int* host = nullptr;
    unsigned int* host_dev = nullptr;
};

namespace mi {
namespace {

constexpr int BACK_CTAS = 296;  // of k_back_act at most: two on an SM

int64_t rows_of(int l, int B) {  // GEMM rows (output voxels × batch) of layer l
    if (l < NCONV) return (int64_t)B * DIM[l + 1] * DIM[l + 1] * DIM[l + 1];
    return B;
}

void free_net(mi_initnet* n) {
    if (!n) return;
    mi_context* ctx = n->ctx;
    for (auto& l : n->L) {
        for (float* p : {l.w, l.b, l.gw, l.gb, l.mw, l.vw, l.mb, l.vb, l.wpart, l.bpart}) dev_free(ctx, p);
        dev_free(ctx, l.wb);
        dev_free(ctx, l.dzb);
    }
    for (auto p : n->col) dev_free(ctx, p);
    for (auto p : n->xb) dev_free(ctx, p);
    dev_free(ctx, n->out);
    dev_free(ctx, n->dcol);
    dev_free(ctx, n->slices);
    pinned_free(ctx, n->host);
    delete n;
}

// BF16 copies of every weight after they were set
cudaError_t refresh_bf16(mi_initnet* n) {
    for (auto& l : n->L) {
        const int64_t cnt = (int64_t)l.out * l.kp;
        k_to_bf16<<<grid1(cnt), 256, 0, n->ctx->stream>>>(l.w, l.wb, cnt);
    }
    return cudaGetLastError();
}

// floats of split-K scratch the GEMM (M, N, K) needs
size_t slice_floats(int M, int N, int K) {
    const int S = k_splits(M, N, K);
    return S > 1 ? (size_t)S * M * N : 0;
}

// Layer l's product, bias and ReLU: rows × kp of x into BF16 activations, or for the last
// layer (no ReLU) FP32 into y.
cudaError_t layer_forward(mi_initnet* n, int l, int B, const __nv_bfloat16* x, float* y) {
    const Layer& L = n->L[l];
    const int M = (int)rows_of(l, B), S = k_splits(M, L.out, L.kp);
    const Operand a{x, L.kp, false}, w{L.wb, L.kp, false};
    __nv_bfloat16* act = n->xb[l];
    if (S == 1)
        return product(n->ctx, M, L.out, L.kp, a, w, tc::Epilogue{y, L.out, L.b, act, L.out, y ? 0 : 1, 0}, 1, n->host_dev);
    const cudaError_t e = product(n->ctx, M, L.out, L.kp, a, w, tc::Epilogue{n->slices, L.out, nullptr, nullptr, 0, 0, 0}, S,
                                  n->host_dev);
    if (e != cudaSuccess) return e;
    const int64_t mn = (int64_t)M * L.out;
    return pdl::launch(k_slices_act, grid1(mn), 256, 0, n->ctx->stream, n->slices, S, mn, L.b, L.out, act);
}

// forward pass of B samples (input x: B × 32³ × 2 FP32, channels-last) into out (B × 12)
cudaError_t forward(mi_initnet* n, int B, const float* x, float* out) {
    cudaStream_t st = n->ctx->stream;
    auto grid = [&](int l) { return dim3((unsigned)((rows_of(l, 1) * (n->L[l].kp / 8) + 255) / 256), (unsigned)std::min(B, 65535)); };
    cudaError_t e = cudaSuccess;
    for (int l = 0; l < NCONV && e == cudaSuccess; ++l) {
        __nv_bfloat16* col = n->col[l];
        switch (l) {
            case 0: e = pdl::launch(k_im2col<DIM[0], CH[0], 64, float>, grid(l), 256, 0, st, x, B, col); break;
            case 1: e = pdl::launch(k_im2col<DIM[1], CH[1], 27 * CH[1], __nv_bfloat16>, grid(l), 256, 0, st, n->xb[0], B, col); break;
            case 2: e = pdl::launch(k_im2col<DIM[2], CH[2], 27 * CH[2], __nv_bfloat16>, grid(l), 256, 0, st, n->xb[1], B, col); break;
            default: e = pdl::launch(k_im2col<DIM[3], CH[3], 27 * CH[3], __nv_bfloat16>, grid(l), 256, 0, st, n->xb[2], B, col); break;
        }
        if (e == cudaSuccess) e = layer_forward(n, l, B, col, nullptr);
    }
    // fc1 on the flattened conv output (B × 1024), fc2 without activation
    if (e == cudaSuccess) e = layer_forward(n, NCONV, B, n->xb[NCONV - 1], nullptr);
    if (e == cudaSuccess) e = layer_forward(n, NCONV + 1, B, n->xb[NCONV], out);
    return e;
}

// The partials of every layer's gradients of the mean squared error against target t
// (B × 12) on the network's last output; loss into the host word.
cudaError_t backward(mi_initnet* n, int B, const float* t) {
    mi_context* ctx = n->ctx;
    cudaStream_t st = ctx->stream;
    Layer& top = n->L[NLAYER - 1];
    cudaError_t e = pdl::launch(k_mse, 1, 256, 0, st, n->out, t, B, FC2_OUT, top.dzb, dz_ld(FC2_OUT), top.bpart,
                                reinterpret_cast<float*>(n->host_dev + 1));
    top.bparts = 1;
    for (int l = NLAYER - 1; l >= 0 && e == cudaSuccess; --l) {
        Layer& L = n->L[l];
        const int rows = (int)rows_of(l, B);
        // the layer's input (BF16, rows × kp): im2col rows or the previous activation
        const __nv_bfloat16* xin = l < NCONV ? n->col[l] : n->xb[l - 1];
        const Operand dz{L.dzb, dz_ld(L.out), false}, dzt{L.dzb, dz_ld(L.out), true};
        // dW (out × kp) = dZᵀ · X, k the rows
        L.wparts = k_splits(L.out, L.kp, rows);
        e = product(ctx, L.out, L.kp, rows, dzt, Operand{xin, L.kp, true},
                    tc::Epilogue{L.wparts > 1 ? L.wpart : L.gw, L.kp, nullptr, nullptr, 0, 0, 0}, L.wparts, n->host_dev);
        if (l == 0 || e != cudaSuccess) break;
        // the gradient of the layer's input (rows × kp) = dZ · W (out is at most four k tiles, so
        // never split)
        e = product(ctx, rows, L.kp, L.out, dz, Operand{L.wb, L.kp, true},
                    tc::Epilogue{n->dcol, L.kp, nullptr, nullptr, 0, 0, 0}, 1, n->host_dev);
        if (e != cudaSuccess) break;
        // back to the previous layer's activations, through its ReLU
        Layer& P = n->L[l - 1];
        const int64_t prows = rows_of(l - 1, B);
        const __nv_bfloat16* act = n->xb[l - 1];
        const int grid = (int)std::min<int64_t>(BACK_CTAS, (prows * (P.out / 4) + 255) / 256);
        P.bparts = grid;
        switch (l) {
            case 1: e = pdl::launch(k_back_act<DIM[1], CH[1], 27 * CH[1]>, grid, 256, 0, st, n->dcol, act, prows, P.dzb, P.bpart); break;
            case 2: e = pdl::launch(k_back_act<DIM[2], CH[2], 27 * CH[2]>, grid, 256, 0, st, n->dcol, act, prows, P.dzb, P.bpart); break;
            case 3: e = pdl::launch(k_back_act<DIM[3], CH[3], 27 * CH[3]>, grid, 256, 0, st, n->dcol, act, prows, P.dzb, P.bpart); break;
            case 4: e = pdl::launch(k_back_act<0, CH[4], 0>, grid, 256, 0, st, n->dcol, act, prows, P.dzb, P.bpart); break;
            default: e = pdl::launch(k_back_act<0, FC1_OUT, 0>, grid, 256, 0, st, n->dcol, act, prows, P.dzb, P.bpart); break;
        }
    }
    return e;
}

// The gradients from their partials and, with lr > 0, the Adam step.
cudaError_t update(mi_initnet* n, float lr) {
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - std::pow(b1, (float)n->step), c2 = 1.0f - std::pow(b2, (float)n->step);
    Tensors T;
    int blocks = 0, k = 0;
    auto add = [&](const Tensor& t) {
        T.t[k] = t;
        T.t[k++].block0 = blocks;
        blocks += tensor_blocks(t.n, t.parts);
    };
    for (const Layer& L : n->L) {
        add(Tensor{L.w, L.gw, L.mw, L.vw, L.wb, L.wparts > 1 ? L.wpart : nullptr, L.out * L.kp, L.wparts, 0});
        add(Tensor{L.b, L.gb, L.mb, L.vb, nullptr, L.bpart, L.out, L.bparts, 0});
    }
    return pdl::launch(k_update, blocks, 256, 0, n->ctx->stream, T, lr, b1, b2, c1, c2, 1e-8f);
}

}  // namespace
}  // namespace mi

extern "C" {

mi_status mi_initnet_create(mi_context* ctx, uint64_t seed, int max_batch, mi_initnet** out) {
    using namespace mi;
    if (!ctx || !out || max_batch < 1) return MI_ERR_INVALID_ARGUMENT;
    MI_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    mi_initnet* n = new (std::nothrow) mi_initnet();
    if (!n) return MI_ERR_OUT_OF_MEMORY;
    n->ctx = ctx;
    n->max_batch = max_batch;
    const int B = max_batch;
    cudaError_t e = cudaSuccess;
    auto alloc = [&](auto** p, size_t bytes) {
        if (e == cudaSuccess) e = dev_alloc(ctx, p, bytes);
        if (e == cudaSuccess) e = cudaMemsetAsync(*p, 0, bytes, ctx->stream);
    };
    // weights: He-uniform from a SplitMix64 stream seeded by `seed`
    uint64_t state = seed;
    auto next_u = [&]() {
        uint64_t z = (state += 0x9E3779B97F4A7C15ull);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (double)(z >> 11) * 0x1p-53;
    };
    size_t max_dcol = 0, max_slices = 0;
    for (int l = 0; l < NLAYER; ++l) {
        Layer& L = n->L[l];
        int fan_in;
        if (l < NCONV) {
            L.out = CH[l + 1];
            L.in = kraw(l);
            L.kp = kpad(l);
        } else if (l == NCONV) {
            L.out = FC1_OUT;
            L.in = L.kp = FC1_IN;
        } else {
            L.out = FC2_OUT;
            L.in = L.kp = FC1_OUT;
        }
        fan_in = L.in;
        const size_t wn = (size_t)L.out * L.kp;
        alloc(&L.w, wn * 4);
        alloc(&L.b, L.out * 4);
        alloc(&L.gw, wn * 4);
        alloc(&L.gb, L.out * 4);
        alloc(&L.mw, wn * 4);
        alloc(&L.vw, wn * 4);
        alloc(&L.mb, L.out * 4);
        alloc(&L.vb, L.out * 4);
        alloc(&L.wb, wn * 2);
        std::vector<float> hw(wn, 0.0f);
        const double bound = std::sqrt(6.0 / fan_in) * (l == NLAYER - 1 ? 0.1 : 1.0);
        for (int o = 0; o < L.out; ++o)
            for (int k = 0; k < L.in; ++k) hw[(size_t)o * L.kp + k] = (float)((2.0 * next_u() - 1.0) * bound);
        if (e == cudaSuccess) e = cudaMemcpyAsync(L.w, hw.data(), wn * 4, cudaMemcpyHostToDevice, ctx->stream);
        // for every batch up to max_batch: the slices of a smaller one may be more, but each
        // holds at least four k tiles
        const int64_t rows = rows_of(l, B);
        const size_t most = std::min<int64_t>(296, std::max<int64_t>(1, (rows + 64 * 4 - 1) / (64 * 4)));
        if (l > 0) max_dcol = std::max(max_dcol, (size_t)rows * L.kp);
        if (l < NLAYER - 1) alloc(&n->xb[l], (size_t)rows * L.out * 2);
        if (l < NCONV) alloc(&n->col[l], (size_t)rows * L.kp * 2);
        alloc(&L.dzb, (size_t)rows * dz_ld(L.out) * 2);
        alloc(&L.wpart, most * wn * 4);
        alloc(&L.bpart, (size_t)BACK_CTAS * L.out * 4);
        for (int q = 1; q <= B; ++q) max_slices = std::max(max_slices, slice_floats((int)rows_of(l, q), L.out, L.kp));
    }
    alloc(&n->slices, std::max<size_t>(max_slices, 1) * 4);
    alloc(&n->dcol, max_dcol * 4);
    alloc(&n->out, (size_t)B * FC2_OUT * 4);
    if (e == cudaSuccess) e = pinned_alloc(ctx, (void**)&n->host, (void**)&n->host_dev);
    if (e == cudaSuccess) n->host[0] = n->host[1] = 0u;
    if (e == cudaSuccess) e = mi::refresh_bf16(n);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) {
        mi::free_net(n);
        return mi::cuda_status(ctx, e, "mi_initnet_create");
    }
    *out = n;
    return MI_OK;
}

mi_status mi_initnet_destroy(mi_initnet* n) {
    if (!n) return MI_ERR_INVALID_ARGUMENT;
    cudaSetDevice(n->ctx->device);
    cudaStreamSynchronize(n->ctx->stream);
    mi::free_net(n);
    return MI_OK;
}

// Layer `which` (0–3 convolutions, 4 fc1, 5 fc2): W as out × in (im2col column order
// for the convolutions) and the bias. grads != 0 reads the last computed gradients.
mi_status mi_initnet_get(mi_initnet* n, int which, int grads, float* w, float* b) {
    if (!n || which < 0 || which >= mi::NLAYER) return MI_ERR_INVALID_ARGUMENT;
    const mi::Layer& L = n->L[which];
    std::vector<float> h((size_t)L.out * L.kp);
    MI_CHECK_CUDA(n->ctx, cudaStreamSynchronize(n->ctx->stream));
    MI_CHECK_CUDA(n->ctx, cudaMemcpy(h.data(), grads ? L.gw : L.w, h.size() * 4, cudaMemcpyDeviceToHost));
    if (w)
        for (int o = 0; o < L.out; ++o) std::memcpy(w + (size_t)o * L.in, h.data() + (size_t)o * L.kp, L.in * 4);
    if (b) MI_CHECK_CUDA(n->ctx, cudaMemcpy(b, grads ? L.gb : L.b, L.out * 4, cudaMemcpyDeviceToHost));
    return MI_OK;
}

mi_status mi_initnet_set(mi_initnet* n, int which, const float* w, const float* b) {
    if (!n || which < 0 || which >= mi::NLAYER || !w || !b) return MI_ERR_INVALID_ARGUMENT;
    mi::Layer& L = n->L[which];
    std::vector<float> h((size_t)L.out * L.kp, 0.0f);
    for (int o = 0; o < L.out; ++o) std::memcpy(h.data() + (size_t)o * L.kp, w + (size_t)o * L.in, L.in * 4);
    MI_CHECK_CUDA(n->ctx, cudaMemcpy(L.w, h.data(), h.size() * 4, cudaMemcpyHostToDevice));
    MI_CHECK_CUDA(n->ctx, cudaMemcpy(L.b, b, L.out * 4, cudaMemcpyHostToDevice));
    cudaError_t e = mi::refresh_bf16(n);
    if (e == cudaSuccess) e = cudaStreamSynchronize(n->ctx->stream);
    if (e != cudaSuccess) return mi::cuda_status(n->ctx, e, "mi_initnet_set");
    return MI_OK;
}

static mi_status check_err(mi_initnet* n, cudaError_t e, const char* where) {
    if (e == cudaSuccess) e = cudaStreamSynchronize(n->ctx->stream);
    if (e != cudaSuccess) return mi::cuda_status(n->ctx, e, where);
    if (n->host[0]) {
        n->host[0] = 0u;
        return mi::set_error(n->ctx, MI_ERR_TIMEOUT, "tensor-core GEMM: an mbarrier wait gave up");
    }
    return MI_OK;
}

// out (device, B × 12) = the network on x (device, B × 32³ × 2 FP32, channels-last)
mi_status mi_initnet_forward(mi_initnet* n, int B, const float* x, float* out) {
    if (!n || B < 1 || B > n->max_batch || !x || !out) return MI_ERR_INVALID_ARGUMENT;
    MI_CHECK_CUDA(n->ctx, cudaSetDevice(n->ctx->device));
    return check_err(n, mi::forward(n, B, x, out), "mi_initnet_forward");
}

// One training step on B samples: forward, mean squared error against t (device,
// B × 12), backward; Adam (β1 0.9, β2 0.999, ε 1e-8) when lr > 0. loss (host) may be NULL.
mi_status mi_initnet_train_step(mi_initnet* n, int B, const float* x, const float* t, float lr, float* loss) {
    using namespace mi;
    if (!n || B < 1 || B > n->max_batch || !x || !t) return MI_ERR_INVALID_ARGUMENT;
    MI_CHECK_CUDA(n->ctx, cudaSetDevice(n->ctx->device));
    cudaError_t e = forward(n, B, x, n->out);
    if (e == cudaSuccess) e = backward(n, B, t);
    if (e == cudaSuccess) {
        if (lr > 0.0f) n->step += 1;
        e = update(n, lr);
    }
    mi_status s = check_err(n, e, "mi_initnet_train_step");
    if (s == MI_OK && loss) std::memcpy(loss, &n->host[1], 4);
    return s;
}

// The network's input for one pair: fixed and moving resampled (linear) onto a 32³ grid
// spanning the fixed image (centre-preserving, spacing · size/32), each normalised to
// zero mean and unit variance, interleaved channels-last into out (device, 32³ × 2).
mi_status mi_initnet_prepare(mi_context* ctx, const mi_image* fixed, const mi_image* moving, float* out) {
    if (!ctx || !fixed || !moving || !out) return MI_ERR_INVALID_ARGUMENT;
    mi_geometry g = fixed->geo;
    for (int d = 0; d < 3; ++d) {
        const double f = (double)fixed->geo.size[d] / 32.0;
        g.size[d] = 32;
        g.spacing[d] = fixed->geo.spacing[d] * f;
    }
    for (int i = 0; i < 3; ++i) {
        double acc = 0.0;
        for (int j = 0; j < 3; ++j) {
            const double delta = ((double)fixed->geo.size[j] - 1.0) / 2.0 - ((double)fixed->geo.size[j] / 32.0) * 31.0 / 2.0;
            acc += fixed->geo.direction[i * 3 + j] * fixed->geo.spacing[j] * delta;
        }
        g.origin[i] = fixed->geo.origin[i] + acc;
    }
    mi_image *rf = nullptr, *rm = nullptr;
    mi_status s = mi_image_resample(ctx, fixed, &g, 0.0, &rf);
    if (s == MI_OK) s = mi_image_resample(ctx, moving, &g, 0.0, &rm);
    if (s == MI_OK) {
        mi::k_normalise<<<1, 256, 0, ctx->stream>>>(rf->data, rf->n, out, 0);
        mi::k_normalise<<<1, 256, 0, ctx->stream>>>(rm->data, rm->n, out, 1);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) s = mi::cuda_status(ctx, e, "mi_initnet_prepare");
    }
    mi_image_free(rf);
    mi_image_free(rm);
    return s;
}

mi_status mi_gemm_bf16_tn(mi_context* ctx, int M, int N, int K, const void* A, int lda, const void* B, int ldb,
                          float* C, int ldc) {
    if (!ctx || M < 1 || N < 1 || K < 1 || !A || !B || !C || lda < K || ldb < K || ldc < N)
        return MI_ERR_INVALID_ARGUMENT;
    MI_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    unsigned int *err = nullptr, *err_dev = nullptr;  // a pinned word and its device address
    cudaError_t e = mi::pinned_alloc(ctx, (void**)&err, (void**)&err_dev);
    if (e == cudaSuccess) *err = 0u;
    // a product whose M × N tiles alone would leave most SMs idle is split over K into
    // partial products summed in slice order, as the network's layers do
    const int S = ldc == N ? mi::k_splits(M, N, K) : 1;
    float* slices = nullptr;
    if (e == cudaSuccess && S > 1) e = mi::dev_alloc(ctx, &slices, (size_t)S * M * N * sizeof(float));
    const auto* a16 = static_cast<const __nv_bfloat16*>(A);
    const auto* b16 = static_cast<const __nv_bfloat16*>(B);
    if (e == cudaSuccess && S > 1) {
        e = mi::gemm_dispatch(ctx, M, N, K, a16, lda, b16, ldb, slices, N, S, err_dev);
        if (e == cudaSuccess) {
            mi::k_sum_slices<<<mi::grid1((int64_t)M * N), 256, 0, ctx->stream>>>(slices, S, (int64_t)M * N, C);
            e = cudaGetLastError();
        }
    } else if (e == cudaSuccess) {
        e = mi::gemm_dispatch(ctx, M, N, K, a16, lda, b16, ldb, C, ldc, 1, err_dev);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    const unsigned int h = err ? *reinterpret_cast<volatile unsigned int*>(err) : 0u;
    mi::dev_free(ctx, slices);
    mi::pinned_free(ctx, err);
    if (e != cudaSuccess) return mi::cuda_status(ctx, e, "mi_gemm_bf16_tn");
    if (h) return mi::set_error(ctx, MI_ERR_TIMEOUT, "tensor-core GEMM: an mbarrier wait gave up");
    return MI_OK;
}

}  // extern "C"
