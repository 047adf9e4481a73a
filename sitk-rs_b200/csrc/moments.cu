// The Mattes metric's shared-sampler siblings behind the same seam: mean squares
// and normalised cross-correlation, as the reference's device metrics compute them
// (registration/device.rs:203-620 DeviceMeanSquaresMetric / DeviceCorrelationMetric;
// cuda/ops/mean_squares.rs, cuda/ops/correlation.rs).
//
// Both are moment reductions: every per-sample term is a product of the sample's
// residual (or shifted values) with the moving gradient and the fixed point, so for any
// global-affine transform, J(x) = J(x_ref) + Σ_e (x − x_ref)_e·C_e, the derivative
// factors through a fixed set of parameter-free moments and the host contracts them
// with the transform's Jacobian form in FP64. Per weight w the moments are
// A_j = Σ w·g_j and B_jm = Σ w·g_j·(idx − mid)_m, g the gradient in index space and idx the
// sample's grid index about the grid's centre (half-integers, exact): the two linear maps
// to physical space (∇M = Mᵀ·g, x − x_ref = M_f·(idx − mid)) are applied once, to the sums.
//
//   mean squares (14 moments; mean_squares.rs:21-44): Σd², count, A and B of w = d = m − f
//     value = Σd² / count,  ∂/∂p_k = 2/count · (Σ_d Jref[d][k]·S0[d] + Σ_de C_e[d][k]·S1[d][e])
//   correlation (42 moments; correlation.rs:31-52): count, Σf′, Σm′, Σf′², Σm′², Σf′m′, A and B of
//     w = f′, m′ and 1, over values shifted by constants, f′ = f − f₀, m′ = m − m₀. With
//     u = f̄ − f₀ and v = m̄ − m₀ the mean-subtracted moments are sff = Σf′² − n·u² and so on, and
//     those of f1 = f′ − u are the f′ ones less u times the unit ones: one pass over the
//     samples instead of one for the means and one for the moments.
//     value = −sfm²/(sff·smm), ∂/∂p_k = −2·sfm/(sff·smm)·(fdm_k − sfm/smm·mdm_k)
//     The shift is formed at set-up, from values spread over the samples and the moving values
//     where the samples lie with the grids' centres put on one another (k_shift).
//     Cancellation costs a factor 1 + n·u²/sff of the rounding; where that passes 2 (an
//     overlap whose mean is more than a standard deviation from the shift) the pass is
//     repeated with the means it found. Against 64 bits the value is off by 0.4–1.4e-15 of
//     itself for overlaps 0 to 95 standard deviations from the moving volume's mean, as with
//     two passes; without the repeats by 1e-14 at 30 and 1.8e-12 at 95.
//
// The sampler is the Mattes metric's: the continuous index from the composite map,
// replaced by the reference's exact chain wherever a decision (inside test, mask
// rounding) or the gradient's cell could differ, so the valid-sample set is the
// reference's exactly. Values, gradients and every accumulator are FP64; each thread
// sums its samples in order, CTAs reduce in a fixed tree and the last CTA folds the
// CTA partials in a fixed order, so a result is bit-identical run to run. Against the
// reference's serial sums the difference is reduction rounding only.
//
// Bound: the latency of index → corners → interpolant at the warps the accumulators leave room
// for (five CTAs of 128 threads on an SM, three for correlation): half of the cycles issue
// and the FP64 pipe is 28 % busy. So a cell's value and gradient are lerps sharing
// their differences (22 FP64 operations; products of corner weights took about 130), floors
// and integer conversions are adds of 2^52-sized constants, the decisions that are not
// near a threshold compare integers. Evaluations: 240×239×155 mean squares 156 → 122 µs, 256³ at 10 %
// correlation 86 → 56 µs and mean squares 51 → 42 µs.
#include <cfloat>
#include <cmath>
#include <cstring>

#include "internal.h"
#include "sampler.cuh"
#include "sampler64.cuh"
#include "eval_device.cuh"
#include "point_map.h"

namespace mi {
void index_to_physical(const mi_geometry& g, double* m);

namespace {

constexpr int MOM_BLOCK = 128;
constexpr int MS_SLOTS = 14;    // Σd², count, A[3], B[9]
constexpr int NCC_SLOTS = 42;   // count, Σf′, Σm′, Σf′², Σm′², Σf′m′, then A[3], B[9] of f′, m′, 1
constexpr int SHIFT_VALUES = 4096;
enum { MODE_MS = 0, MODE_NCC = 1 };

template <int MODE, bool GRAD>
__host__ __device__ constexpr int slots() {
    return MODE == MODE_MS ? (GRAD ? MS_SLOTS : 2) : (GRAD ? NCC_SLOTS : 6);
}

struct MomArgs {
    const float* moving;       // the moving volume, x-fastest
    const float* fixed;        // each sample's fixed value, in sample order (the fixed volume
                               // itself when every voxel is a sample)
    const uint8_t* mmask;
    const uint32_t* samples;   // flat indices in brick order, or null for the whole grid
    uint32_t n;
    double* partials;          // [slots][grid]
    unsigned int* counter;     // arrivals of the current launch (reset by the last CTA)
    double* result_host;       // mapped host mirror the last CTA writes
    unsigned long long seq;    // the evaluation's number
    const double* shift;       // f₀, m₀ (correlation; by value in the arguments: 65 µs for 55 at 256³)
    FracWords words;
    double mid[3];             // the fixed grid's centre in index units
};

// A sample's place in the moving volume: the cell, the fractions, and the grid index.
struct Place {
    int cell[3];
    double fr[3], idx[3];
};

// The decisions of a sample that is not certainly in the volume's interior, or not
// certainly off a cell face: those of prep_fast with the exact chain where they could flip.
template <bool GRAD>
__device__ __noinline__ bool locate_edge(const SamplerParams& P, uint32_t i, uint32_t j, uint32_t k, double* c, int* cell) {
    const double ce = P.cerr;
    bool need = false;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (!(c[d] >= P.ilo && c[d] < P.ihi[d])) {
            if (c[d] < P.olo || c[d] >= P.ohi[d]) return false;
            need = true;
        }
        const double f = c[d] - floor(c[d]);
        // the interpolant's gradient jumps across cell faces: take the reference's cell
        if (GRAD && (f <= ce || f >= 1.0 - ce)) need = true;
        if (P.has_mmask) {
            const double h = c[d] + 0.5;
            if (floor(h - ce) != floor(h + ce)) need = true;
        }
    }
    if (need) {
        exact_index(P, i, j, k, c);
#pragma unroll
        for (int d = 0; d < 3; ++d)
            if (!(c[d] >= -0.5 && c[d] < P.mhi[d])) return false;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) cell[d] = (int)floor(c[d]);
    return true;
}

// False when the sample maps outside the moving buffer or onto a masked voxel
// (MovingImage::value_and_physical_gradient, registration/metric.rs:795-861).
template <bool GRAD>
__device__ __forceinline__ bool locate(const SamplerParams& P, const MomArgs& a, uint32_t flat, Place& p) {
    uint32_t i, j, k;
    grid_index(P, flat, i, j, k);
    p.idx[0] = u32_to_f64(i);
    p.idx[1] = u32_to_f64(j);
    p.idx[2] = u32_to_f64(k);
    double c[3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
        c[r] = fma(P.cA[r * 3 + 2], p.idx[2], fma(P.cA[r * 3 + 1], p.idx[1], fma(P.cA[r * 3], p.idx[0], P.cb[r])));
    const int st = place64<GRAD>(P, a.words, c, p.cell, p.fr);
    if (st == SAMPLE_OFF) return false;
    if (st == SAMPLE_UNSURE) {
        // (copies: what a call takes by address lives in memory, here only on this path)
        double e[3] = {c[0], c[1], c[2]};
        int cell[3];
        if (!locate_edge<GRAD>(P, i, j, k, e, cell)) return false;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            p.cell[d] = cell[d];
            p.fr[d] = e[d] - floor(e[d]);
        }
        return !P.has_mmask || mask_exact(P, a.mmask, e);
    }
    return !P.has_mmask || mask64(P, a.mmask, p.cell, p.fr);
}

// acc[0..2] += w·g, acc[3 + 3j + m] += w·g_j·x_m
__device__ __forceinline__ void add_moments(double* acc, double w, const double* g, const double* x) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const double wg = w * g[j];
        acc[j] += wg;
#pragma unroll
        for (int m = 0; m < 3; ++m) acc[3 + j * 3 + m] = fma(wg, x[m], acc[3 + j * 3 + m]);
    }
}

template <int MODE, bool GRAD>
constexpr int moment_blocks() { return !GRAD ? 8 : (MODE == MODE_NCC ? 3 : 5); }

// AHEAD: the next sample is requested before the current one is finished. Worth its registers
// with the derivative, whose accumulators leave few warps to wait with (256³ correlation
// 53 against 57 µs, mean squares of a 50 % list 120 against 127), except for mean squares
// over the whole grid, whose loads are coalesced (113 against 120 µs without); not for
// the value alone.
// WEIGHTED: the interpolant as the reference sums it, for a volume with infinite voxels.
template <int MODE, bool GRAD, bool AHEAD, bool WEIGHTED = false>
__global__ void __launch_bounds__(MOM_BLOCK, (moment_blocks<MODE, GRAD>()))
k_moments(const __grid_constant__ SamplerParams P, const MomArgs a) {
    constexpr int NS = slots<MODE, GRAD>(), PAD = (NS + 15) / 16 * 16, NW = MOM_BLOCK / 32;
    double acc[PAD];
#pragma unroll
    for (int q = 0; q < PAD; ++q) acc[q] = 0.0;
    uint32_t count = 0;
    const double f0 = MODE == MODE_NCC ? a.shift[0] : 0.0, m0 = MODE == MODE_NCC ? a.shift[1] : 0.0;
    const uint32_t stride = gridDim.x * blockDim.x;
    uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    auto index_of = [&](uint32_t t) { return t < a.n ? (a.samples ? __ldg(a.samples + t) : t) : 0u; };
    // a sample's place, corners and fixed value, requested
    struct Ahead {
        Place p;
        float v[8], f;
        bool ok;
    };
    auto request = [&](uint32_t t, uint32_t flat, Ahead& q) {
        q.ok = t < a.n && locate<GRAD>(P, a, flat, q.p);
        if (q.ok) {
            load_corners(P, a.moving, q.p.cell, q.v);
            q.f = __ldg(a.fixed + t);
        }
    };
    auto finish = [&](const Ahead& q) {
        if (!q.ok) return;
        const double fv = (double)q.f;
        double g[3], x[3];
        const double mv = WEIGHTED ? interpolate_weighted<GRAD>(q.v, q.p.fr, g) : interpolate<GRAD>(q.v, q.p.fr, g);
        if (GRAD) {
#pragma unroll
            for (int m = 0; m < 3; ++m) x[m] = q.p.idx[m] - a.mid[m];
        }
        ++count;
        if (MODE == MODE_MS) {
            const double diff = mv - fv;
            acc[0] = fma(diff, diff, acc[0]);
            if (GRAD) add_moments(acc + 2, diff, g, x);
        } else {
            const double f1 = fv - f0, m1 = mv - m0;
            acc[1] += f1;
            acc[2] += m1;
            acc[3] = fma(f1, f1, acc[3]);
            acc[4] = fma(m1, m1, acc[4]);
            acc[5] = fma(f1, m1, acc[5]);
            if (GRAD) {
                add_moments(acc + 6, f1, g, x);
                add_moments(acc + 18, m1, g, x);
                add_moments(acc + 30, 1.0, g, x);
            }
        }
    };
    uint32_t flat = index_of(s);
    if (AHEAD) {
        Ahead next;
        request(s, flat, next);
        flat = index_of(s + stride);
        while (s < a.n) {
            const Ahead cur = next;
            s += stride;
            request(s, flat, next);
            flat = index_of(s + stride);
            finish(cur);
        }
    } else {
        for (; s < a.n; s += stride) {
            Ahead cur;
            const uint32_t here = flat;
            flat = index_of(s + stride);
            request(s, here, cur);
            finish(cur);
        }
    }
    acc[MODE == MODE_MS ? 1 : 0] = (double)count;

    // The CTA's sums. Over a warp, sixteen slots at a time: each xor step halves the slots a
    // lane keeps, so lanes 2t and 2t + 1 end with slot t (16 shuffles for 16 slots).
    __shared__ double red[NW][PAD];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < PAD; q += 16) {
        int slot = q;
#pragma unroll
        for (int h = 8, off = 16; h >= 1; h >>= 1, off >>= 1) {
            const bool hi = (lane & off) != 0;
#pragma unroll
            for (int t = 0; t < h; ++t) {
                const double keep = hi ? acc[q + t + h] : acc[q + t];
                const double give = hi ? acc[q + t] : acc[q + t + h];
                acc[q + t] = keep + __shfl_xor_sync(0xffffffffu, give, off);
            }
            slot += hi ? h : 0;
        }
        acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], 1);
        if ((lane & 1) == 0) red[warp][slot] = acc[q];
    }
    __syncthreads();
    for (int q = threadIdx.x; q < NS; q += MOM_BLOCK) {
        double t = red[0][q];
#pragma unroll
        for (int w = 1; w < NW; ++w) t += red[w][q];
        a.partials[(size_t)q * gridDim.x + blockIdx.x] = t;
    }
    if (!last_to_arrive(a.counter)) return;
    // Fold in a fixed order: lane l of slot q's warp turn sums the partials of CTAs l, l + 32, …
    // (eight loads issued together), then an xor tree; one warp a slot.
    for (int q = warp; q < NS; q += NW) {
        const double* src = a.partials + (size_t)q * gridDim.x;
        double t = 0.0;
        for (unsigned int b0 = lane; b0 < gridDim.x; b0 += 8 * 32) {
            double u[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) u[e] = b0 + e * 32 < gridDim.x ? __ldcg(src + b0 + e * 32) : 0.0;
#pragma unroll
            for (int e = 0; e < 8; ++e) t += u[e];
        }
        t = slice_sum(t);
        if (lane == 0) {
            red[0][q] = t;
            a.result_host[q] = t;
        }
    }
    if (threadIdx.x == 0) *a.counter = 0u;
    __syncthreads();
    // the tag that lets the host take the moments without waiting for the stream (publish_seq's:
    // the words may arrive in any order)
    if (warp == 0) {
        unsigned long long h = 0ull;
        for (int q = lane; q < NS; q += 32) h ^= publish_word(q, (unsigned long long)__double_as_longlong(red[0][q]));
#pragma unroll
        for (int off = 16; off; off >>= 1) h ^= __shfl_xor_sync(0xffffffffu, h, off);
        if (lane == 0)
            *reinterpret_cast<volatile unsigned long long*>(a.result_host + NCC_SLOTS) = h ^ publish_mix(a.seq);
    }
}

// The shift of correlation's values, near the means of whatever part of the images an
// evaluation will see: up to SHIFT_VALUES samples look for the moving voxel nearest to them
// under P's map, in the volume and the mask; the means of those that find one and of what
// they find, or, where fewer than one in eight does, of all of them and of voxels spread
// over the moving volume. Values that are not finite are passed over; 0 where there is none.
constexpr int SHIFT_BLOCK = 1024;
__global__ void __launch_bounds__(SHIFT_BLOCK)
k_shift(const __grid_constant__ SamplerParams P, const float* __restrict__ fixed, const uint32_t* __restrict__ samples,
        int64_t n, const float* __restrict__ moving, const uint8_t* __restrict__ mmask, int64_t nm,
        double* __restrict__ shift, double* __restrict__ host) {
    __shared__ double red[32];
    double f = 0.0, m = 0.0, mine = 0.0, all = 0.0, nall = 0.0;  // of samples that find a voxel; of all of them
    auto take = [&](uint32_t at) {
        const float v = __ldg(moving + at);
        if ((mmask && !__ldg(mmask + at)) || !isfinite(v)) return false;
        m += (double)v;
        mine += 1.0;
        return true;
    };
    const int64_t count = min(n, (int64_t)SHIFT_VALUES);
    for (int64_t q = threadIdx.x; q < count; q += SHIFT_BLOCK) {
        const int64_t s = q * (n / count);
        const float v = __ldg(fixed + s);
        uint32_t i, j, k, at = 0;
        grid_index(P, samples ? __ldg(samples + s) : (uint32_t)s, i, j, k);
        bool inside = true;
        for (int r = 0; r < 3; ++r) {
            const double c = floor(fma(P.cA[r * 3 + 2], (double)k, fma(P.cA[r * 3 + 1], (double)j, fma(P.cA[r * 3], (double)i, P.cb[r]))) + 0.5);
            inside = inside && c >= 0.0 && c < (double)P.msz[r];
            if (inside) at += (uint32_t)c * (r == 0 ? 1u : (r == 1 ? P.ms1 : P.ms2));
        }
        if (!isfinite(v)) continue;
        all += (double)v;
        nall += 1.0;
        if (inside && take(at)) f += (double)v;
    }
    double nm1 = block_sum(mine, red), nf = nm1;
    f = block_sum(f, red);
    all = block_sum(all, red);
    nall = block_sum(nall, red);
    if (nm1 * 8.0 < (double)count) {
        f = all;
        nf = nall;
        m = mine = 0.0;
        const int64_t spread = min(nm, (int64_t)SHIFT_VALUES);
        for (int64_t q = threadIdx.x; q < spread; q += SHIFT_BLOCK) take((uint32_t)(q * (nm / spread)));
        nm1 = block_sum(mine, red);
    }
    m = block_sum(m, red);
    if (threadIdx.x == 0) {
        host[0] = shift[0] = nf > 0.0 ? f / nf : 0.0;
        host[1] = shift[1] = nm1 > 0.0 ? m / nm1 : 0.0;
    }
}

// Each sample's fixed value, gathered once: the fixed image and the samples do not
// change over the metric's life, so the evaluations read them contiguously instead of
// gathering from the whole fixed volume.
__global__ void k_gather_fixed(const float* __restrict__ fixed, const uint32_t* __restrict__ samples, int64_t n,
                               float* __restrict__ out) {
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < n; s += (int64_t)gridDim.x * blockDim.x)
        out[s] = fixed[samples[s]];
}

template <int MODE, bool GRAD>
int grid_of(mi_context* ctx, int64_t n) {
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_moments<MODE, GRAD, GRAD>, MOM_BLOCK, 0) != cudaSuccess)
        cudaGetLastError();
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + MOM_BLOCK - 1) / MOM_BLOCK, (int64_t)ctx->num_sms * std::max(occ, 1)));
}

}  // namespace

mi_status moments_setup(mi_metric* m, const float* fixed) {
    mi_context* ctx = m->ctx;
    MomentsWs& w = m->mom;
    const int64_t n = m->n_samples;
    const bool ncc = m->metric_kind == MI_METRIC_CORRELATION;
    w.grid = ncc ? grid_of<MODE_NCC, false>(ctx, n) : grid_of<MODE_MS, false>(ctx, n);
    w.grid_grad = ncc ? grid_of<MODE_NCC, true>(ctx, n) : grid_of<MODE_MS, true>(ctx, n);
    cudaStream_t st = ctx->stream;
    MI_CHECK_CUDA(ctx, dev_alloc(ctx, &w.partials, (size_t)std::max(w.grid, w.grid_grad) * NCC_SLOTS * sizeof(double)));
    MI_CHECK_CUDA(ctx, dev_alloc(ctx, &w.shift, 4 * sizeof(double)));
    MI_CHECK_CUDA(ctx, dev_alloc(ctx, &w.counter, sizeof(unsigned int)));
    MI_CHECK_CUDA(ctx, cudaMemsetAsync(w.counter, 0, sizeof(unsigned int), st));
    if (m->samples && m->n_samples > 0) {
        MI_CHECK_CUDA(ctx, dev_alloc(ctx, &w.fval, (size_t)m->n_samples * sizeof(float)));
        const int g = (int)std::max<int64_t>(1, std::min<int64_t>((m->n_samples + 255) / 256, (int64_t)ctx->num_sms * 8));
        k_gather_fixed<<<g, 256, 0, st>>>(fixed, m->samples, m->n_samples, w.fval);
        MI_CHECK_CUDA(ctx, cudaGetLastError());
    }
    static_assert((NCC_SLOTS + 1) * sizeof(double) <= PINNED_BLOCK, "the moments' mirror is one pinned block");
    MI_CHECK_CUDA(ctx, pinned_alloc(ctx, reinterpret_cast<void**>(&w.host), reinterpret_cast<void**>(&w.host_dev)));
    if (ncc) {
        // the map that puts the centres of the grids on one another
        SamplerParams P = m->base;
        double stage[12] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
        double mm[9];
        index_to_physical(m->mgeo, mm);
        for (int d = 0; d < 3; ++d) {
            stage[9 + d] = P.morigin[d] - P.xref[d];
            for (int e = 0; e < 3; ++e) stage[9 + d] += mm[d * 3 + e] * 0.5 * (double)(m->mgeo.size[e] - 1);
        }
        pm_stages(P, stage, 1);
        pm_compose(P);
        const int64_t nm = m->mgeo.size[0] * m->mgeo.size[1] * m->mgeo.size[2];
        k_shift<<<1, SHIFT_BLOCK, 0, st>>>(P, w.fval ? w.fval : fixed, m->samples, n, m->moving, m->mmask, nm, w.shift,
                                          w.host_dev);
        MI_CHECK_CUDA(ctx, cudaGetLastError());
        MI_CHECK_CUDA(ctx, cudaStreamSynchronize(st));
        w.base[0] = w.host[0];
        w.base[1] = w.host[1];
    }
    std::memset(w.host, 0, (NCC_SLOTS + 1) * sizeof(double));  // no stale tag
    return MI_OK;
}

void moments_free(mi_metric* m) {
    mi_context* ctx = m->ctx;
    MomentsWs& w = m->mom;
    dev_free(ctx, w.partials);
    dev_free(ctx, w.shift);
    dev_free(ctx, w.counter);
    dev_free(ctx, w.fval);
    pinned_free(ctx, w.host);
    w = MomentsWs{};
}

// One pass over the samples with the shift at `shift`; its ns moments in m->mom.host.
// `weighted` (mean squares): see k_moments.
static mi_status moments_pass(mi_metric* m, const SamplerParams& P, const double* shift, bool grad, int ns,
                              bool weighted = false) {
    mi_context* ctx = m->ctx;
    MomentsWs& w = m->mom;
    Workspace& ws = m->ws;
    cudaStream_t st = ctx->stream;
    MomArgs a;
    a.moving = m->moving;
    a.fixed = w.fval ? w.fval : m->fixed;
    a.mmask = m->mmask;
    a.samples = m->samples;
    a.n = (uint32_t)m->n_samples;
    a.partials = w.partials;
    a.counter = w.counter;
    a.result_host = w.host_dev;
    a.seq = ++ws.seq;
    a.shift = shift;
    a.words = frac_words(P.cerr);
    for (int d = 0; d < 3; ++d) a.mid[d] = (double)P.xmid[d];
    const bool timing = ws.timing != 0;
    if (timing) MI_CHECK_CUDA(ctx, cudaEventRecord(ws.ev[0], st));
    const int grid = grad ? w.grid_grad : w.grid;
    if (m->metric_kind == MI_METRIC_CORRELATION) {
        if (grad)
            k_moments<MODE_NCC, true, true><<<grid, MOM_BLOCK, 0, st>>>(P, a);
        else
            k_moments<MODE_NCC, false, false><<<grid, MOM_BLOCK, 0, st>>>(P, a);
    } else {
        if (weighted && grad)
            k_moments<MODE_MS, true, false, true><<<grid, MOM_BLOCK, 0, st>>>(P, a);
        else if (weighted)
            k_moments<MODE_MS, false, false, true><<<grid, MOM_BLOCK, 0, st>>>(P, a);
        else if (grad && m->samples)
            k_moments<MODE_MS, true, true><<<grid, MOM_BLOCK, 0, st>>>(P, a);
        else if (grad)
            k_moments<MODE_MS, true, false><<<grid, MOM_BLOCK, 0, st>>>(P, a);
        else
            k_moments<MODE_MS, false, false><<<grid, MOM_BLOCK, 0, st>>>(P, a);
    }
    MI_CHECK_CUDA(ctx, cudaGetLastError());
    if (timing) {
        MI_CHECK_CUDA(ctx, cudaEventRecord(ws.ev[4], st));
        MI_CHECK_CUDA(ctx, cudaStreamSynchronize(st));
        float t = 0.f;
        MI_CHECK_CUDA(ctx, cudaEventElapsedTime(&t, ws.ev[0], ws.ev[4]));
        ws.ms[0] += t;
        return MI_OK;
    }
    // wait for the published tag (evaluate(), mattes.cu)
    const volatile unsigned long long* words = reinterpret_cast<const volatile unsigned long long*>(w.host);
    auto published = [&]() {
        unsigned long long h = publish_mix(a.seq);
        for (int q = 0; q < ns; ++q) h ^= publish_word(q, words[q]);
        return words[NCC_SLOTS] == h;
    };
    for (uint32_t spin = 1;; ++spin) {
        if (published()) return MI_OK;
        if ((spin & 63u) == 0u) {
            const cudaError_t q = cudaStreamQuery(st);
            if (q == cudaSuccess) {
                if (published()) return MI_OK;
                return set_error(ctx, MI_ERR_CUDA, "the evaluation finished without publishing its result");
            }
            if (q != cudaErrorNotReady) return cuda_status(ctx, q, "cudaStreamQuery");
        }
    }
}

mi_status evaluate_moments(mi_metric* m, const SamplerParams& P, const double* jac0, const double* jacc, int nparams,
                           bool want_derivative, double* value, double* derivative, int64_t* valid) {
    mi_context* ctx = m->ctx;
    MomentsWs& w = m->mom;
    const bool ncc = m->metric_kind == MI_METRIC_CORRELATION;
    const int ns = ncc ? (want_derivative ? NCC_SLOTS : 6) : (want_derivative ? MS_SLOTS : 2);
    mi_status s = moments_pass(m, P, w.shift, want_derivative, ns);
    if (s != MI_OK) return s;
    const double* r = w.host;
    // Not a number: a voxel that is not, or an infinite one, whose mean square is +inf. The pass
    // again with the weighted sum tells them apart (a test of every sample's value in the pass
    // itself: 122.5 -> 124.5 µs at 240×239×155). Correlation is NaN of either.
    if (!ncc && std::isnan(r[0])) {
        s = moments_pass(m, P, w.shift, want_derivative, ns, true);
        if (s != MI_OK) return s;
    }
    // The moments A[j], B[j][m] in physical space: S0 = Mᵀ·A, S1[d][e] = Σ_jm M[j][d]·B[j][m]·M_f[e][m];
    // then the contraction with J(x) = J(x_ref) + Σ_e (x − x_ref)_e·C_e.
    double jref[3 * MI_MAX_PARAMS];
    if (want_derivative)
        for (int i = 0; i < 3 * nparams; ++i) {
            double v = jac0[i];
            for (int e = 0; e < 3; ++e) v += P.xref[e] * jacc[e * 3 * nparams + i];
            jref[i] = v;
        }
    auto contract = [&](const double* A, double* out) {
        const double* B = A + 3;
        double s0[3], s1[9];
        for (int d = 0; d < 3; ++d) {
            s0[d] = A[0] * P.mp2i[d] + A[1] * P.mp2i[3 + d] + A[2] * P.mp2i[6 + d];
            double t[3];
            for (int q = 0; q < 3; ++q) t[q] = B[q] * P.mp2i[d] + B[3 + q] * P.mp2i[3 + d] + B[6 + q] * P.mp2i[6 + d];
            for (int e = 0; e < 3; ++e)
                s1[d * 3 + e] = t[0] * P.fi2p[e * 3] + t[1] * P.fi2p[e * 3 + 1] + t[2] * P.fi2p[e * 3 + 2];
        }
        for (int k = 0; k < nparams; ++k) {
            double gk = 0.0;
            for (int d = 0; d < 3; ++d) {
                gk += jref[d * nparams + k] * s0[d];
                for (int e = 0; e < 3; ++e) gk += jacc[e * 3 * nparams + d * nparams + k] * s1[d * 3 + e];
            }
            out[k] = gk;
        }
    };
    if (m->ws.timing) m->ws.timed_evals += 1;
    if (want_derivative)
        for (int k = 0; k < nparams; ++k) derivative[k] = 0.0;
    if (!ncc) {
        // registration/cuda.rs:381-412 (contract)
        const double count = r[1];
        if (valid) *valid = (int64_t)count;
        if (count == 0.0) {
            *value = DBL_MAX;
            return MI_OK;
        }
        if (!want_derivative) {
            *value = r[0] / count;  // mean_squares_value divides
            return MI_OK;
        }
        const double inv = 1.0 / count;
        *value = r[0] * inv;
        contract(r + 2, derivative);
        for (int k = 0; k < nparams; ++k) derivative[k] = 2.0 * derivative[k] * inv;
        return MI_OK;
    }
    // registration/cuda.rs:439-490 (contract_correlation), on the shifted moments
    const double count = r[0];
    if (valid) *valid = (int64_t)count;
    if (count == 0.0) {
        *value = DBL_MAX;
        return MI_OK;
    }
    double u = r[1] / count, v = r[2] / count;
    double sff = r[3] - count * u * u, smm = r[4] - count * v * v;
    if (count * u * u > sff || count * v * v > smm) {
        // the shift is far from the means: again with the means themselves
        const double means[2] = {w.base[0] + u, w.base[1] + v};
        MI_CHECK_CUDA(ctx, cudaMemcpyAsync(w.shift + 2, means, sizeof(means), cudaMemcpyHostToDevice, ctx->stream));
        s = moments_pass(m, P, w.shift + 2, want_derivative, ns);
        if (s != MI_OK) return s;
        u = r[1] / count;
        v = r[2] / count;
        sff = r[3] - count * u * u;
        smm = r[4] - count * v * v;
    }
    const double sfm = r[5] - count * u * v;
    const double m2f2 = smm * sff;
    if (!(m2f2 > DBL_EPSILON) && m2f2 == m2f2) {
        *value = DBL_MAX;
        return MI_OK;
    }
    *value = -sfm * sfm / m2f2;
    if (want_derivative) {
        double fd[MI_MAX_PARAMS], md[MI_MAX_PARAMS], gd[MI_MAX_PARAMS];
        contract(r + 6, fd);
        contract(r + 18, md);
        contract(r + 30, gd);
        for (int k = 0; k < nparams; ++k) {
            const double fdm = fd[k] - u * gd[k], mdm = md[k] - v * gd[k];
            derivative[k] = -2.0 * sfm / (sff * smm) * (fdm - sfm / smm * mdm);
        }
    }
    return MI_OK;
}

}  // namespace mi
