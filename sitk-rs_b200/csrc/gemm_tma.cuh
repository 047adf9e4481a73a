// The tensor-core product of gemm_tc.cuh for operands that TMA can read (leading
// dimensions a multiple of eight, 16-byte aligned bases):
//
//     C[M×N] = A[M×K] · B[N×K]ᵀ     (BF16 operands, K contiguous, FP32 accumulation)
//
// A persistent CTA of six warps per SM walks the work items (128 × NT tile of C, K slice):
//   warp 0  one lane requests A and B tiles of 64 k (128-byte rows, 128-byte swizzle) into
//           a ring of shared-memory stages, as far ahead as the ring goes
//   warp 1  one lane issues four tcgen05.mma per stage into one of two accumulators in
//           tensor memory and commits the stage back to warp 0 (MT = 2: eight, one accumulator)
//   warps 2–5  read the other accumulator (tcgen05.ld, 32 rows a warp) and store 32 × 32
//           blocks by TMA from shared memory, two in flight a warp
// so copies, products and stores of neighbouring items overlap. Rows, columns and k past
// the operands' ends arrive as zeros. Every element's products are accumulated in k
// order, as in gemm_tc.cuh: same bits.
//
// Bound: a 128 × 256 tile brings 48 KB from L2 for 2·128·256·64 operations, so 148 CTAs ask it
// for more than it gives (12 TB/s seen) before the tensor pipe is full; with MT = 2 a CTA
// takes two blocks of 128 rows on one B tile, 64 KB for twice the operations, and one
// accumulator (of 512 columns) instead of two. Narrow products (NT ≤ 64) are bound by the
// bytes of A. 4096³ with warm caches: 109 µs a call with two blocks (1,263 TFLOP/s, 0.77 of the
// measured 1,646), 118 with one (126 and 134 with cold inputs); the one-stage kernel of gemm_tc.cuh took 1,489 µs. Products of few k are
// bound by their output: 32,768 × 432 × 32 writes 57 MB in 18 µs by TMA stores, 32 µs when
// the four warps turned the blocks in shared memory and stored rows themselves (290
// instructions a block).
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
#include "pdl.cuh"

namespace mi {
namespace tc {

constexpr int TMA_THREADS = 192;
constexpr unsigned int TMA_POLLS = 1u << 20;  // of mbarrier.try_wait, each suspending up to 2 µs

// MT: blocks of 128 rows in a tile, one or two.
template <int NT, int MT = 1>
struct TmaShape {
    static constexpr uint32_t A_BYTES = MT * TILE_M * TILE_K * 2, B_BYTES = NT * TILE_K * 2;
    static constexpr uint32_t STAGE = A_BYTES + B_BYTES;
    static constexpr uint32_t EPI = 4 * 2 * 32 * 32 * 4;  // four warps' 32 × 32 blocks, two each
    static constexpr int FIT = (int)((225 * 1024 - EPI) / STAGE);
    static constexpr int STAGES = FIT < 8 ? FIT : 8;
    static constexpr uint32_t BARS = STAGES * STAGE + EPI;
    static constexpr uint32_t SMEM = BARS + (2 * STAGES + 5) * 8 + 1024;  // and the alignment of the base
    static constexpr int ACCS = MT == 1 ? 2 : 1;                          // accumulators of MT · NT columns
    static constexpr uint32_t COLS = 2 * NT < 32 ? 32 : 2 * NT;           // all of them, a power of two
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

// ReLU whose sign bit says whether z was positive: 0 for a z so small that BF16 rounds it to
// zero, −0 for one that is not positive (or NaN). −0 counts as 0 wherever it is used.
__device__ __forceinline__ float relu(float z) { return z > 0.f ? z : -0.f; }

// What becomes of an element z of the product: stored in C, or where that is null as BF16 in
// X; z + bias[column] with a bias (the layers' widths are multiples of four), then relu()
// when relu is set. Splits store the plain partial products in C. With
// `tma` the blocks leave by TMA through the output's map: pitch and base multiples of 16
// bytes. X always goes that way.
struct Epilogue {
    float* C;
    int ldc;
    const float* bias;
    __nv_bfloat16* X;
    int ldx;
    int relu;
    int tma;
};

// 16-byte chunk q of row `row` in a block of rows of ROW bytes, by TMA's swizzle of that width
template <int ROW>
__device__ __forceinline__ uint32_t block_chunk(int row, int q) {
    static_assert(ROW == 32 || ROW == 64 || ROW == 128, "");
    const int x = ROW == 128 ? row & 7 : (ROW == 64 ? (row >> 1) & 3 : (row >> 2) & 1);
    return (uint32_t)(row * ROW + ((q ^ x) << 4));
}
__device__ __forceinline__ void st_shared16(uint32_t at, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void tma_store(const CUtensorMap* map, uint32_t src, int col, int row, int z) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(map), "r"(src),
                 "r"(col), "r"(row), "r"(z)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// Work item `item`: K slices slowest, then columns, rows fastest (CTAs that run together
// share a B tile and the A tiles stay in L2).
struct Item {
    int m0, n0, z, kt0, kt1;
};
template <int NT, int MT>
__device__ __forceinline__ Item item_at(int item, int mt, int nt, int ktiles, int per) {
    Item w;
    w.m0 = (item % mt) * (MT * TILE_M);
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

template <int NT, bool A_KROWS, bool B_KROWS, int MT = 1>
__global__ void __launch_bounds__(TMA_THREADS, 1)
k_gemm_tma(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
           const __grid_constant__ CUtensorMap mapOut, int M, int N, int K, const Epilogue E, int splits, unsigned int* err) {
    static_assert(!B_KROWS || NT % 64 == 0, "k-rows tiles come in boxes of 64");
    static_assert(MT == 1 || (!A_KROWS && 2 * NT <= 512), "two blocks of rows fill the tensor memory");
    using S = TmaShape<NT, MT>;
    constexpr uint32_t ACCS = S::ACCS;
    extern __shared__ uint8_t raw[];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int quit;
    const uint32_t base = (smem_u32(raw) + 1023u) & ~1023u;
    const uint32_t epi = base + S::STAGES * S::STAGE, bars = base + S::BARS;
    const uint32_t full = bars, empty = bars + S::STAGES * 8, tfull = bars + S::STAGES * 16, tempty = tfull + 16,
                   drained = tempty + 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl::launch_dependents();
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
    pdl::wait_previous();

    const int mt = (M + MT * TILE_M - 1) / (MT * TILE_M), nt = (N + NT - 1) / NT;
    const int ktiles = (K + TILE_K - 1) / TILE_K, per = (ktiles + splits - 1) / splits;
    const int items = mt * nt * splits;

    if (warp == 0) {
        if (lane == 0) {
            uint32_t count = 0;  // tiles requested
            bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
                const Item w = item_at<NT, MT>(it, mt, nt, ktiles, per);
                for (int kt = w.kt0; kt < w.kt1; ++kt, ++count) {
                    const uint32_t s = count % S::STAGES, round = count / S::STAGES;
                    if (!bar_wait(empty + s * 8, (round & 1) ^ 1, &quit)) {
                        ok = false;
                        break;
                    }
                    const uint32_t dst = base + s * S::STAGE;
                    bar_expect(full + s * 8, S::STAGE);
                    request_tile<TILE_M, A_KROWS>(dst, &mapA, full + s * 8, kt * TILE_K, w.m0);
                    if (MT == 2)
                        request_tile<TILE_M, A_KROWS>(dst + TILE_M * TILE_K * 2, &mapA, full + s * 8, kt * TILE_K, w.m0 + TILE_M);
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
                const Item w = item_at<NT, MT>(it, mt, nt, ktiles, per);
                if (w.kt0 >= w.kt1) continue;  // an empty slice has no product
                const uint32_t a = tiles % ACCS;
                if (!bar_wait(tempty + a * 8, ((tiles / ACCS) & 1) ^ 1, &quit)) break;
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
                    for (int qh = 0; qh < TILE_K / 16 * MT; ++qh) {
                        const int q = qh / MT, h = qh % MT;  // both blocks of rows for each of B's 16 k
                        const uint32_t acc = (kt > w.kt0 || q > 0) ? 1u : 0u;
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
                            "}" ::"r"(tmem + (a * MT + h) * NT),
                            "l"(ad + h * (TILE_M * TILE_K * 2 >> 4) + q * A_STEP), "l"(bd + q * B_STEP), "r"(idesc), "r"(acc));
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
        const uint32_t blocks = epi + (warp - 2) * 2 * 4096;
        float* block = reinterpret_cast<float*>(raw + (blocks - smem_u32(raw)));
        const int ldc = E.ldc;
        uint32_t tiles = 0, stored = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x) {
            const Item w = item_at<NT, MT>(it, mt, nt, ktiles, per);
            const bool any = w.kt0 < w.kt1;
            const uint32_t a = tiles % ACCS;
            if (any) {
                if (!__all_sync(0xffffffffu, bar_wait(tfull + a * 8, (tiles / ACCS) & 1, &quit))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            constexpr int W = NT < 32 ? NT : 32;  // columns a block
#pragma unroll 1
            for (int ch = 0; ch < MT * NT; ch += W) {
                const int c0 = ch % NT, row0 = w.m0 + (ch / NT) * TILE_M + quad * 32;
                uint32_t r[W];
                if (any) {
                    const uint32_t at = tmem + ((uint32_t)(quad * 32) << 16) + a * (MT * NT) + ch;
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
                    if (ch + W >= MT * NT) {  // the accumulator has been read
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        if (lane == 0) bar_arrive(tempty + a * 8);
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < W; ++q) r[q] = 0u;
                }
                const int col0 = w.n0 + c0;
                if (col0 >= N || row0 >= M) continue;
                if (E.bias) {
#pragma unroll
                    for (int q = 0; q < W; q += 4) {
                        if (col0 + q >= N) break;
                        const float4 b = __ldca(reinterpret_cast<const float4*>(E.bias + col0 + q));
                        const float add[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const float v = __uint_as_float(r[q + k]) + add[k];
                            r[q + k] = __float_as_uint(E.relu ? relu(v) : v);
                        }
                    }
                }
                if (E.tma) {
                    // the block of two stores ago has been read
                    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    __syncwarp();
                    const uint32_t at = blocks + (stored++ & 1) * 4096;
                    if (E.C) {
#pragma unroll
                        for (int q = 0; q < W / 4; ++q)
                            st_shared16(at + block_chunk<W * 4>(lane, q), r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
                    } else {
                        uint32_t h[W / 2];
#pragma unroll
                        for (int q = 0; q < W / 2; ++q) {
                            const __nv_bfloat162 v =
                                __floats2bfloat162_rn(__uint_as_float(r[2 * q]), __uint_as_float(r[2 * q + 1]));
                            h[q] = *reinterpret_cast<const uint32_t*>(&v);
                        }
#pragma unroll
                        for (int q = 0; q < W / 8; ++q)
                            st_shared16(at + block_chunk<W * 2>(lane, q), h[4 * q], h[4 * q + 1], h[4 * q + 2], h[4 * q + 3]);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) tma_store(&mapOut, at, col0, row0, w.z);
                } else {
                    // any pitch and base: each row's columns by the lanes in turn
#pragma unroll
                    for (int q = 0; q < W; q += 4)
                        *reinterpret_cast<uint4*>(block + lane * 36 + q) = make_uint4(r[q], r[q + 1], r[q + 2], r[q + 3]);
                    __syncwarp();
                    float* out = E.C + ((size_t)w.z * M + row0) * ldc + col0;
                    if (lane < W && col0 + lane < N)
#pragma unroll 8
                        for (int i = 0; i < 32; ++i)
                            if (row0 + i < M) out[(size_t)i * ldc + lane] = block[i * 36 + lane];
                    __syncwarp();
                }
            }
            if (any) ++tiles;
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // its memory is read, C written
    }
    __syncthreads();
    if (threadIdx.x == 0 && quit) *reinterpret_cast<volatile unsigned int*>(err) = 1u;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::COLS));
}

}  // namespace tc
}  // namespace mi
