// The tensor-core product of gemm_tc.cuh for operands that TMA can read (leading
// dimensions a multiple of eight, 16-byte aligned bases):
//
//     C[M×N] = A[M×K] · B[N×K]ᵀ     (BF16 operands, K contiguous, FP32 accumulation)
//
// A persistent CTA of six warps per SM walks the work items (128 × NT tile of C, K slice):
//   warp 0  one lane requests A and B tiles of 64 k (128-byte rows, 128-byte swizzle) into
//           a ring of shared-memory stages, as far ahead as the ring goes
//   warp 1  one lane issues four tcgen05.mma per stage into one of two accumulators in
//           tensor memory and commits the stage back to warp 0
//   warps 2–5  read the other accumulator (tcgen05.ld, 32 rows a warp), turn 32 × 32
//           blocks in shared memory and store whole 128-byte rows of C
// so copies, products and stores of neighbouring items overlap. Rows, columns and k past
// the operands' ends arrive as zeros. Every element's products are accumulated in k
// order, as in gemm_tc.cuh: same bits.
//
// Bound: a 128 × 256 tile does 2·128·256·64 operations for 48 KB brought in and 48 KB read
// by the tensor core, so shared-memory bandwidth and the tensor pipe are close; the ring
// (four stages) covers L2's latency. Narrow products (NT ≤ 64) are bound by the bytes of A.
// 4096³: 137 µs a call (1,005 TFLOP/s, 0.63 of 1.59 PFLOP/s; four rounds of CTAs for 3.46
// rounds of tiles); the one-stage kernel of gemm_tc.cuh took 1,489 µs.
//
// An operand may also be stored the other way round, k slowest ("k-rows": element (r, k) at
// k·ld + r, as a product's transpose needs it): its tiles come as boxes of 64 rows × 64 k
// and the instruction reads them MN-major, so nothing is transposed beforehand.
//
// Every wait is bounded: a role that gives up raises *err (a word the host can read, so the
// call needs no copy back) and leaves, the others follow
// (their own waits see the flag), the copies in flight are waited for and the tensor
// memory is freed.
#pragma once

#include <cuda.h>

#include "gemm_tc.cuh"

namespace mi {
namespace tc {

constexpr int TMA_THREADS = 192;
constexpr unsigned int TMA_POLLS = 1u << 20;  // of mbarrier.try_wait, each suspending up to 2 µs

template <int NT>
struct TmaShape {
    static constexpr uint32_t A_BYTES = TILE_M * TILE_K * 2, B_BYTES = NT * TILE_K * 2;
    static constexpr uint32_t STAGE = A_BYTES + B_BYTES;
    static constexpr uint32_t EPI = 4 * 32 * 36 * 4;  // four warps' 32 × 32 blocks, rows of 36 floats
    static constexpr int FIT = (int)((220 * 1024 - EPI) / STAGE);
    static constexpr int STAGES = FIT < 8 ? FIT : 8;
    static constexpr uint32_t BARS = STAGES * STAGE + EPI;
    static constexpr uint32_t SMEM = BARS + (2 * STAGES + 5) * 8 + 1024;  // and the alignment of the base
    static constexpr uint32_t COLS = 2 * NT < 32 ? 32 : 2 * NT;           // two accumulators, a power of two
};

__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 2000;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t"
        "}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
// Waits for the phase of that parity; false when it gave up or another role did.
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, volatile int* quit) {
    for (unsigned int polls = 0; polls < TMA_POLLS; ++polls) {
        if (bar_try(bar, parity)) return true;
        if (*quit) return false;
    }
    *quit = 1;
    return false;
}
__device__ __forceinline__ void tma_tile(uint32_t dst, const CUtensorMap* map, uint32_t bar, int k, int row) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
            "r"(dst),
        "l"(map), "r"(bar), "r"(k), "r"(row)
        : "memory");
}

// shared-memory matrix descriptor of a K-major tile with 128-byte rows and the 128-byte
// swizzle: 1024 bytes from one group of eight rows to the next, layout type 2 at bit 61
__device__ __forceinline__ uint64_t swizzled_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

// The same of an MN-major tile (boxes of 64 rows × 64 k: 128-byte lines of 64 rows, one k
// each): 8192 bytes from one 64 rows to the next, 1024 from eight k to the next.
__device__ __forceinline__ uint64_t swizzled_desc_mn(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(8192 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
           (2ull << 61);
}

// What becomes of an element z of the product: stored in C (where not null), and with X as
// BF16 of z + bias[column], negative values cut off when relu is set. With a bias C gets
// z + bias. Splits store the plain partial products.
struct Epilogue {
    float* C;
    int ldc;
    const float* bias;
    __nv_bfloat16* X;
    int ldx;
    int relu;
};

// Work item `item`: K slices slowest, then columns, rows fastest (CTAs that run together
// share a B tile and the A tiles stay in L2).
struct Item {
    int m0, n0, z, kt0, kt1;
};
template <int NT>
__device__ __forceinline__ Item item_at(int item, int mt, int nt, int ktiles, int per) {
    Item w;
    w.m0 = (item % mt) * TILE_M;
    w.n0 = (item / mt) % nt * NT;
    w.z = item / (mt * nt);
    w.kt0 = min(ktiles, w.z * per);
    w.kt1 = min(ktiles, w.kt0 + per);
    return w;
}

// `rows` rows from `row` at 64 k from `k` into dst.
template <int ROWS, bool KROWS>
__device__ __forceinline__ void request_tile(uint32_t dst, const CUtensorMap* map, uint32_t bar, int k, int row) {
    if (!KROWS) {
        tma_tile(dst, map, bar, k, row);
    } else {
#pragma unroll
        for (int r = 0; r < ROWS; r += 64) tma_tile(dst + r * 128, map, bar, row + r, k);
    }
}

template <int NT, bool A_KROWS, bool B_KROWS>
__global__ void __launch_bounds__(TMA_THREADS, 1)
k_gemm_tma(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, int M, int N, int K,
           const Epilogue E, int splits, unsigned int* __restrict__ err) {
    static_assert(!B_KROWS || NT % 64 == 0, "k-rows tiles come in boxes of 64");
    using S = TmaShape<NT>;
    extern __shared__ uint8_t raw[];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int quit;
    const uint32_t base = (smem_u32(raw) + 1023u) & ~1023u;
    const uint32_t epi = base + S::STAGES * S::STAGE, bars = base + S::BARS;
    const uint32_t full = bars, empty = bars + S::STAGES * 8, tfull = bars + S::STAGES * 16, tempty = tfull + 16,
                   drained = tempty + 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < S::STAGES; ++s) {
            bar_init(full + s * 8, 1);
            bar_init(empty + s * 8, 1);
        }
        for (int a = 0; a < 2; ++a) {
            bar_init(tfull + a * 8, 1);
            bar_init(tempty + a * 8, 4);
        }
        bar_init(drained, 1);
        quit = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(S::COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    const int mt = (M + TILE_M - 1) / TILE_M, nt = (N + NT - 1) / NT;
    const int ktiles = (K + TILE_K - 1) / TILE_K, per = (ktiles + splits - 1) / splits;
    const int items = mt * nt * splits;

    if (warp == 0) {
        if (lane == 0) {
            uint32_t count = 0;  // tiles requested
            bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
                const Item w = item_at<NT>(it, mt, nt, ktiles, per);
                for (int kt = w.kt0; kt < w.kt1; ++kt, ++count) {
                    const uint32_t s = count % S::STAGES, round = count / S::STAGES;
                    if (!bar_wait(empty + s * 8, (round & 1) ^ 1, &quit)) {
                        ok = false;
                        break;
                    }
                    const uint32_t dst = base + s * S::STAGE;
                    bar_expect(full + s * 8, S::STAGE);
                    request_tile<TILE_M, A_KROWS>(dst, &mapA, full + s * 8, kt * TILE_K, w.m0);
                    request_tile<NT, B_KROWS>(dst + S::A_BYTES, &mapB, full + s * 8, kt * TILE_K, w.n0);
                }
            }
            if (!ok) {
                // the copies in flight write into this CTA's memory: let them land
                for (uint32_t c = count > (uint32_t)S::STAGES ? count - S::STAGES : 0; c < count; ++c)
                    for (unsigned int polls = 0; polls < TMA_POLLS; ++polls)
                        if (bar_try(full + (c % S::STAGES) * 8, (c / S::STAGES) & 1)) break;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            // bits 15 and 16: A and B are MN-major
            const uint32_t idesc = instr_desc(TILE_M, NT) | (A_KROWS ? 1u << 15 : 0u) | (B_KROWS ? 1u << 16 : 0u);
            // sixteen k further: 32 bytes inside the swizzled rows, or two groups of eight k
            constexpr uint64_t A_STEP = A_KROWS ? 2048 >> 4 : 32 >> 4, B_STEP = B_KROWS ? 2048 >> 4 : 32 >> 4;
            uint32_t count = 0, tiles = 0;
            bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
                const Item w = item_at<NT>(it, mt, nt, ktiles, per);
                if (w.kt0 >= w.kt1) continue;  // an empty slice has no product
                const uint32_t a = tiles & 1;
                if (!bar_wait(tempty + a * 8, ((tiles >> 1) & 1) ^ 1, &quit)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int kt = w.kt0; kt < w.kt1; ++kt, ++count) {
                    const uint32_t s = count % S::STAGES;
                    if (!bar_wait(full + s * 8, (count / S::STAGES) & 1, &quit)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t at = base + s * S::STAGE, bt = at + S::A_BYTES;
                    const uint64_t ad = A_KROWS ? swizzled_desc_mn(at) : swizzled_desc(at);
                    const uint64_t bd = B_KROWS ? swizzled_desc_mn(bt) : swizzled_desc(bt);
#pragma unroll
                    for (int q = 0; q < TILE_K / 16; ++q) {
                        const uint32_t acc = (kt > w.kt0 || q > 0) ? 1u : 0u;
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
                            "}" ::"r"(tmem + a * NT),
                            "l"(ad + q * A_STEP), "l"(bd + q * B_STEP), "r"(idesc), "r"(acc));
                    }
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                     empty + s * 8)
                                 : "memory");
                }
                if (!ok) break;
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 tfull + a * 8)
                             : "memory");
                ++tiles;
            }
            if (quit) {  // the products in flight read this CTA's memory: let them end
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(drained)
                             : "memory");
                for (unsigned int polls = 0; polls < TMA_POLLS; ++polls)
                    if (bar_try(drained, 0)) break;
            }
        }
        __syncwarp();
    } else {
        const int quad = warp & 3;  // the tensor-memory lanes this warp can read
        float* block = reinterpret_cast<float*>(raw + (epi - smem_u32(raw))) + (warp - 2) * 32 * 36;
        const int ldc = E.ldc;
        const bool vec = (ldc & 3) == 0 && ((uintptr_t)E.C & 15) == 0;
        uint32_t tiles = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x) {
            const Item w = item_at<NT>(it, mt, nt, ktiles, per);
            const bool any = w.kt0 < w.kt1;
            const uint32_t a = tiles & 1;
            if (any) {
                if (!__all_sync(0xffffffffu, bar_wait(tfull + a * 8, (tiles >> 1) & 1, &quit))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            float* out = E.C + (size_t)w.z * M * ldc;
            constexpr int W = NT < 32 ? NT : 32;  // columns a block
            const int row0 = w.m0 + quad * 32;
#pragma unroll 1
            for (int c0 = 0; c0 < NT; c0 += W) {
                uint32_t r[W];
                if (any) {
                    const uint32_t at = tmem + ((uint32_t)(quad * 32) << 16) + a * NT + c0;
#pragma unroll
                    for (int q = 0; q < W; q += 16)
                        asm volatile(
                            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
                            "%13, %14, %15}, [%16];"
                            : "=r"(r[q]), "=r"(r[q + 1]), "=r"(r[q + 2]), "=r"(r[q + 3]), "=r"(r[q + 4]), "=r"(r[q + 5]),
                              "=r"(r[q + 6]), "=r"(r[q + 7]), "=r"(r[q + 8]), "=r"(r[q + 9]), "=r"(r[q + 10]),
                              "=r"(r[q + 11]), "=r"(r[q + 12]), "=r"(r[q + 13]), "=r"(r[q + 14]), "=r"(r[q + 15])
                            : "r"(at + q));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (c0 + W >= NT) {  // the accumulator has been read
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        if (lane == 0) bar_arrive(tempty + a * 8);
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < W; ++q) r[q] = 0u;
                }
                if (w.n0 + c0 >= N) continue;
#pragma unroll
                for (int q = 0; q < W; q += 4)
                    *reinterpret_cast<uint4*>(block + lane * 36 + q) = make_uint4(r[q], r[q + 1], r[q + 2], r[q + 3]);
                __syncwarp();
                constexpr int PER_ROW = W / 4, ROWS = 32 / PER_ROW;  // lanes a row, rows at once
                const int q = (lane % PER_ROW) * 4, col = w.n0 + c0 + q;
#pragma unroll
                for (int i = 0; i < 32; i += ROWS) {
                    const int rr = i + lane / PER_ROW, row = row0 + rr;
                    if (row < M) {
                        float4 v = *reinterpret_cast<const float4*>(block + rr * 36 + q);
                        float* dst = out + (size_t)row * ldc + col;
                        if (E.bias && col + 4 <= N) {  // the layers' widths are multiples of four
                            const float4 b = __ldg(reinterpret_cast<const float4*>(E.bias + col));
                            v = make_float4(v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w);
                            if (E.X) {
                                if (E.relu) v = make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
                                const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
                                *reinterpret_cast<uint2*>(E.X + (size_t)row * E.ldx + col) =
                                    make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
                            }
                        }
                        if (!E.C) {
                        } else if (vec && col + 4 <= N) {
                            *reinterpret_cast<float4*>(dst) = v;
                        } else {
                            if (col < N) dst[0] = v.x;
                            if (col + 1 < N) dst[1] = v.y;
                            if (col + 2 < N) dst[2] = v.z;
                            if (col + 3 < N) dst[3] = v.w;
                        }
                    }
                }
                __syncwarp();
            }
            if (any) ++tiles;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && quit) *reinterpret_cast<volatile unsigned int*>(err) = 1u;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::COLS));
}

}  // namespace tc
}  // namespace mi
