// Batched registration: many pairs of uneven sizes advance one optimizer iteration
// per pass of two launches — the histogram pass over every active pair's chunks, then
// the tail and derivative pass over the same chunks, in which the CTA that finishes a
// pair makes its optimizer step — with all optimizer state on the device. A pass is captured in a CUDA graph
// (several passes per graph) and replayed until every pair has stopped; the host
// only reads how many pairs are still active after each replay.
//
// Per pair the arithmetic is the single-pair path's: the same sampler, histogram,
// tail and moment code (eval_device.cuh), the same regular-step gradient descent
// (rsgd.h) and the same point-map constants (point_map.h). What differs is the
// launch shape: a pair's samples are cut into chunks of `chunk` samples, whose moments are
// summed chunk by chunk, the CTAs take equal shares of the active pairs' samples and
// chunks, and the fixed-point unit of the histogram follows from the chunk size, so
// values agree with the single-pair path to that unit.
//
// The chunk size and the number of privatised histogram copies are chosen by a small
// autotuner that times the candidates on the batch itself and caches the choice per
// (bins, sample-count class).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <tuple>
#include <vector>

#include "eval_device.cuh"
#include "internal.h"
#include "point_map.h"
#include "rsgd.h"

namespace mi {
mi_status shift_corners(int kind, const double* params, int nparams, const double* fixed, int nfixed,
                        const mi_geometry& fg, rsgd::Corners& c);
}  // namespace mi

namespace mi {
namespace {

// What is left of a pair: nothing once it has stopped. Two lists: the first is read by the
// histogram pass and cleared, entry by entry, by the steps in the derivative pass; that
// pass reads the second, the histogram pass's copy, so that no list changes under its readers.
struct Work {
    unsigned int samples;  // rounded up to UNIT
    unsigned int chunks;   // derivative chunks
};
constexpr unsigned int UNIT = 128;          // samples: a histogram share starts on whole 512-byte lines
constexpr unsigned int LEAST_SHARE = 1024;  // samples a histogram CTA takes at least, two a thread

struct PairDev {
    SamplerParams P;
    JacobianForm J;
    EvalArgs a;
    rsgd::Corners corners;
    rsgd::State state;
    double scales[MI_MAX_PARAMS];
    double params[MI_MAX_PARAMS];
    double center[3];
    double value;
    double valid;
    int kind, nparams, nchunks;
    int active;
    int evaluations;
    unsigned int done;  // derivative chunks of this pair finished in the current pass
    unsigned long long stop_ns;  // device global timer when the pair stopped (0: running)
};

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// The device global timer into *t (one thread): the start and end marks of a run.
__global__ void k_stamp(unsigned long long* t) { *t = global_ns(); }

// The next point map of an affine or translation family (transforms.cpp: the
// AffineTransform offset center + t − A·center, mat_vec from 0.0; a translation is
// the identity matrix with the translation as offset).
__device__ void family_stage(int kind, const double* p, const double* center, double* stage) {
    using rsgd::add;
    using rsgd::mul;
    using rsgd::sub;
    if (kind == MI_TRANSFORM_TRANSLATION) {
        for (int i = 0; i < 9; ++i) stage[i] = (i % 4 == 0) ? 1.0 : 0.0;
        for (int d = 0; d < 3; ++d) stage[9 + d] = p[d];
        return;
    }
    for (int i = 0; i < 9; ++i) stage[i] = p[i];
    for (int r = 0; r < 3; ++r) {
        double acc = 0.0;
        for (int c = 0; c < 3; ++c) acc = add(acc, mul(p[r * 3 + c], center[c]));
        stage[9 + r] = sub(add(center[r], p[9 + r]), acc);
    }
}

// What a chunk's samples read of its pair, in shared memory (every pointer and constant would
// otherwise be fetched from global memory again after each store).
struct PairShared {
    alignas(16) unsigned char params[sizeof(SamplerParams)];
    alignas(16) unsigned char args[sizeof(EvalArgs)];
    __device__ SamplerParams& P() { return *reinterpret_cast<SamplerParams*>(params); }
    __device__ const EvalArgs& a() const { return *reinterpret_cast<const EvalArgs*>(args); }
};
__device__ __forceinline__ void copy_words(void* dst, const void* src, size_t bytes) {
    const unsigned int* s = static_cast<const unsigned int*>(src);
    unsigned int* d = static_cast<unsigned int*>(dst);
    for (int i = threadIdx.x; i < (int)(bytes / 4); i += blockDim.x) d[i] = s[i];
}
static_assert(sizeof(SamplerParams) % 4 == 0 && sizeof(EvalArgs) % 4 == 0, "whole words");

// The whole CTA.
__device__ __forceinline__ void load_pair(const PairDev& pd, PairShared& sh) {
    copy_words(sh.params, &pd.P, sizeof(SamplerParams));
    copy_words(sh.args, &pd.a, sizeof(EvalArgs));
    __syncthreads();
}

// Positions along the pairs' remaining work, one after another: the whole CTA computes the
// prefix sums of `key` over the pairs (thread t a run of consecutive ones), and locate()
// finds the pair under a position.
struct Line {
    unsigned long long total;
    unsigned long long first;  // of this thread's run
    int lo, hi;                // the run
};
template <class Key>
__device__ __forceinline__ Line lay_out(const Work* work, int npairs, Key key) {
    __shared__ unsigned long long sums[32];
    const int per = (npairs + (int)blockDim.x - 1) / (int)blockDim.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Line l;
    l.lo = min(npairs, (int)threadIdx.x * per);
    l.hi = min(npairs, l.lo + per);
    unsigned long long own = 0;
    for (int p = l.lo; p < l.hi; ++p) own += key(work[p]);
    unsigned long long scan = own;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const unsigned long long o = __shfl_up_sync(0xffffffffu, scan, off);
        if (lane >= off) scan += o;
    }
    if (lane == 31) sums[warp] = scan;
    __syncthreads();
    unsigned long long before = 0, total = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
        if (w < warp) before += sums[w];
        total += sums[w];
    }
    l.first = before + scan - own;
    l.total = total;
    return l;
}
struct Place {
    int pair;
    unsigned long long start;  // the pair's first position
};
// at < l.total; the whole CTA
template <class Key>
__device__ __forceinline__ Place locate(const Work* work, const Line& l, unsigned long long at, Key key) {
    __shared__ Place found;
    __syncthreads();  // the last one was read
    unsigned long long x = l.first;
    for (int p = l.lo; p < l.hi; ++p) {
        const unsigned long long n = key(work[p]);
        if (at >= x && at - x < n) found = Place{p, x};
        x += n;
    }
    __syncthreads();
    return found;
}

// The histograms of every active pair. Integer sums, so any split of the samples gives the
// same counts: the active pairs' samples are laid end to end and every CTA takes an equal
// share, pair by pair, in segments short enough for the fixed-point unit (seg_max). A
// pass of 24 pairs, 2.45 M samples: 55 µs; 61 µs with whole chunks of 4,096 in turn (610
// over 296 CTAs, so three rounds for 2.06).
__global__ void __launch_bounds__(HIST_BLOCK, HIST_MIN_BLOCKS)
k_batch_hist(PairDev* __restrict__ pairs, Work* __restrict__ work, int npairs, unsigned int seg_max,
             uint32_t* __restrict__ exq) {
    extern __shared__ __align__(16) unsigned int sh[];
    __shared__ PairShared sp;
    pdl::launch_dependents();
    pdl::wait_previous();
    // this CTA's queue for the exact chain: a segment at a time, so at most its samples
    const ExactQueue q{MI_EXACT_DEFERRED ? exq + (size_t)blockIdx.x * seg_max : nullptr, seg_max};
    const auto samples = [](const Work& w) { return w.samples; };
    const Line line = lay_out(work, npairs, samples);
    if (blockIdx.x == 0)  // the derivative pass's copy
        for (int p = threadIdx.x; p < npairs; p += blockDim.x) work[npairs + p] = work[p];
    unsigned long long share = (line.total + gridDim.x - 1) / gridDim.x;
    share = max((share + UNIT - 1) / UNIT * UNIT, (unsigned long long)LEAST_SHARE);
    const unsigned long long end = min(line.total, share * (blockIdx.x + 1));
    for (unsigned long long at = share * blockIdx.x; at < end;) {
        const Place pl = locate(work, line, at, samples);
        const PairDev& pd = pairs[pl.pair];
        load_pair(pd, sp);
        const uint32_t n = sp.a().n;
        const uint32_t first = (uint32_t)(at - pl.start);
        const uint32_t last = (uint32_t)(min(pl.start + (n + UNIT - 1) / UNIT * UNIT, end) - pl.start);
        const uint32_t len = last - first, segs = (len + seg_max - 1) / seg_max;
        const uint32_t seg = ((len + segs - 1) / segs + UNIT - 1) / UNIT * UNIT;  // seg_max is a multiple of UNIT
        for (uint32_t b = first; b < last; b += seg) {
            const uint32_t e = min(min(b + seg, last), n);
            if (b < e) hist_phase<true>(sp.P(), sp.a(), sh, SampleRange{b, e, threadIdx.x & ~31u, blockDim.x}, q);
            __syncthreads();
        }
        at = pl.start + last;
    }
}

// The optimizer's part of a pair, staged for one thread.
struct StepShared {
    rsgd::State state;
    double scaled[MI_MAX_PARAMS], params[MI_MAX_PARAMS], center[3], cmax;
    int go;
};

// The optimizer's decision on the evaluation just made, then the next point map, by the CTA
// that finished the pair's derivative, on copies in shared memory: one thread decides, the
// divisions and the point map's bound are spread (9.6 µs with all of it by one thread,
// 10–14 µs as a launch of its own of one thread a pair). P is that CTA's copy of the
// pair's constants.
__device__ void step_pair(PairDev& pd, Work& work, SamplerParams& P, const mi_rsgd_config& cfg, unsigned int* active_count) {
    __shared__ StepShared s;
    const int np = pd.nparams;
    copy_words(&s.state, &pd.state, sizeof(rsgd::State));
    if ((int)threadIdx.x < np) {
        s.scaled[threadIdx.x] = rsgd::div(pd.a.result[2 + threadIdx.x], pd.scales[threadIdx.x]);
        s.params[threadIdx.x] = pd.params[threadIdx.x];
    }
    if (threadIdx.x < 3) s.center[threadIdx.x] = pd.center[threadIdx.x];
    __syncthreads();
    if (threadIdx.x == 0) {
        pd.evaluations += 1;
        pd.value = pd.a.result[0];
        pd.valid = pd.a.result[1];
        s.go = rsgd::after_scaled(s.state, cfg, pd.corners, s.scaled, s.params) ? 0 : 1;
        if (s.go) {
            double stage[12];
            family_stage(pd.kind, s.params, s.center, stage);
            pm_stages(P, stage, 1);
        } else {
            pd.active = 0;
            work = Work{0u, 0u};
            pd.stop_ns = global_ns();
            atomicSub(active_count, 1u);
        }
    }
    __syncthreads();
    copy_words(&pd.state, &s.state, sizeof(rsgd::State));
    if (s.go) {
        // point_map_fill, the corners in one warp beside the composite map
        if (threadIdx.x == 0) pm_compose(P);
        if (threadIdx.x >= 32 && threadIdx.x < 64) {
            double m = pm_corner(P, threadIdx.x & 7);
#pragma unroll
            for (int off = 4; off; off >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, off));
            if (threadIdx.x == 32) s.cmax = m;
        }
        __syncthreads();
        if (threadIdx.x == 0) pm_bounds(P, s.cmax);
        __syncthreads();
        if ((int)threadIdx.x < np) pd.params[threadIdx.x] = s.params[threadIdx.x];
        copy_words(&pd.P, &P, sizeof(SamplerParams));
    }
}

// A pair whose last chunk this CTA finished.
struct Finished {
    int pair;
    TailCtx t;
};
constexpr int FINISHED_MAX = 4;

// The tail and derivative of every active pair's chunks; with STEP the CTA that finishes a
// pair also makes its optimizer step. A chunk's FP32 sums are its own, whoever forms them:
// every CTA takes an equal run of consecutive chunks, so that a pair's table (k_deriv's,
// stream_table: one round of requests and two barriers) is formed once for all of its
// chunks here, and folds and steps the pairs it finished after its chunks, not between
// them (up to FINISHED_MAX of them waiting). 24 pairs, 610 chunks: 40 µs; 65 µs with a tail
// for every chunk, the steps a launch of their own.
template <bool STEP>
__global__ void __launch_bounds__(DERIV_BLOCK, DERIV_MIN_BLOCKS)
k_batch_deriv(PairDev* __restrict__ pairs, Work* __restrict__ work, int npairs, unsigned int chunk, mi_rsgd_config cfg,
              unsigned int* __restrict__ active_count) {
    extern __shared__ double dsh[];
    __shared__ PairShared sp;
    __shared__ Finished done[FINISHED_MAX];
    __shared__ bool last;
    pdl::launch_dependents();
    pdl::wait_previous();
    // a pair's table weighs about as much as a chunk: its first position is the table's
    const auto chunks = [](const Work& w) { return w.chunks ? w.chunks + 1u : 0u; };
    const Work* left = work + npairs;
    const Line line = lay_out(left, npairs, chunks);
    const unsigned long long begin = line.total * blockIdx.x / gridDim.x, end = line.total * (blockIdx.x + 1) / gridDim.x;
    int nfinished = 0, loaded = -1;
    auto finish = [&]() {
        for (int k = 0; k < nfinished; ++k) {
            const int p = done[k].pair;
            PairDev& pd = pairs[p];
            if (p != loaded) load_pair(pd, sp);
            loaded = p;
            __threadfence();  // the other CTAs' moments and value slices
            const EvalArgs& a = sp.a();
            static_assert(DERIV_BLOCK >= 18 * NMOM + 32, "deriv_fold's value warp");
            deriv_fold<true>(sp.P(), pd.J, a, done[k].t, a.partials, (unsigned int)pd.nchunks);
            if (threadIdx.x == 0) pd.done = 0u;
            const int B = sp.P().bins, nb = B * B + 2 * B;  // joint, counts, column sums
            for (int i = threadIdx.x; i < nb; i += blockDim.x) a.ghist[i] = 0ull;
            __syncthreads();
            if (STEP) step_pair(pd, work[p], sp.P(), cfg, active_count);
            __syncthreads();
        }
        nfinished = 0;
    };
    Place pl{-1, 0ull};
    TableCtx tab;
    unsigned int count = 0, mine = 0;  // the pair's chunks, and those done here
    for (unsigned long long c = begin; c < end; ++c) {
        const bool fresh = pl.pair < 0 || c - pl.start > count;
        if (fresh) {
            pl = locate(left, line, c, chunks);
            if (c == pl.start && ++c == end) break;  // the first position is no chunk
            count = (unsigned int)pairs[pl.pair].nchunks;
            load_pair(pairs[pl.pair], sp);
            loaded = pl.pair;
        }
        const EvalArgs& a = sp.a();
        const unsigned int local = (unsigned int)(c - pl.start) - 1u, first = local * chunk;
        const uint32_t gend = a.n - first <= chunk ? a.npad >> 2 : (first + chunk) >> 2;
        const GroupWork w{first >> 2, gend, threadIdx.x, blockDim.x, a.partials + local, (int64_t)count, (int)local, (int)count};
        RecordGroup cur;
        if (fresh)
            tab = stream_table<GridRecords>(sp.P(), a, dsh, w, cur);
        else if (w.begin + w.first < w.end)
            load_group(a, w.begin + w.first, cur);
        stream_rows<GridRecords>(sp.P(), a, dsh, w, cur, tab);
        ++mine;
        __syncthreads();
        if (c + 1 < end && local + 1 < count) continue;
        // the pair's chunks here are done: with them the pair, if no other CTA has more to come
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            last = atomicAdd(&pairs[pl.pair].done, mine) + mine == count;
            if (last) done[nfinished] = Finished{pl.pair, tab.t};
        }
        mine = 0;
        __syncthreads();
        if (last && ++nfinished == FINISHED_MAX) {
            finish();
            pl.pair = -1;  // the table and the pair's constants may be another's now
        }
    }
    finish();
}

// Autotuner cache: (bins, log2 of the total sample count) → (chunk, coarse copies).
std::mutex g_tune_mu;
std::map<std::pair<int, int>, std::pair<int, int>> g_tune;

}  // namespace
}  // namespace mi

struct mi_batch {
    mi::Held ctx;
    int npairs = 0, bins = 0, kind = 0, nparams = 0;
    std::vector<mi_metric*> metrics;
    std::vector<std::vector<double>> fixed_params;
    std::vector<mi::PairDev> host;  // host mirror of the device pair array
    mi::PairDev* d_pairs = nullptr;
    mi::Work* d_work = nullptr;   // two lists
    int nchunks = 0;
    unsigned int seg_max = 0;     // samples a histogram CTA may add before it flushes
    double* d_partials = nullptr;
    size_t partials_cap = 0;      // doubles
    unsigned int* d_active = nullptr;
    unsigned int* h_active = nullptr;  // pinned
    unsigned long long* d_marks = nullptr;  // device global timer at the start and end of the last run
    uint32_t* d_exq = nullptr;              // per-CTA queues of samples for the exact chain
    size_t exq_len = 0;
    std::vector<double> pair_seconds;       // per pair: start of the last run to its stop
    int grid_hist = 0, grid_deriv = 0;
    int chunk = 0, copies = 0, fine_copies = 0;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int graph_passes = 0;
    mi_rsgd_config graph_cfg{};
};

namespace mi {
namespace {

// The copies alone, by which their number is chosen, and with the column sums after them.
size_t batch_hist_copies(int B, int copies, int fine) {
    return ((size_t)copies * hist_copy_stride(B) + (size_t)fine * hist_fine_stride(B)) * sizeof(unsigned int);
}
size_t batch_hist_smem(int B, int copies, int fine) { return hist_region_bytes(B, copies, fine); }

void release_graph(mi_batch* b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
    b->graph_passes = 0;
}

// Lays out the chunk list and the per-pair histogram units for a (chunk, copies)
// shape, and uploads the pair array.
mi_status shape_batch(mi_batch* b, int chunk, int copies) {
    mi_context* ctx = b->ctx;
    const int B = b->bins;
    int fine = std::max(1, copies / 2);
    while (fine > 1 && batch_hist_copies(B, copies, fine) > 52 * 1024) fine >>= 1;
    if (batch_hist_copies(B, copies, fine) > 200 * 1024)
        return set_error(ctx, MI_ERR_INVALID_ARGUMENT, "histogram copies do not fit in shared memory");
    int nchunks = 0, per_thread_max = 1 << 20;
    int64_t total = 0;
    size_t poff = 0;
    for (int p = 0; p < b->npairs; ++p) {
        mi_metric* m = b->metrics[p];
        const uint32_t n = (uint32_t)m->n_samples;
        const int nc = std::max<int>(1, (int)((n + chunk - 1) / chunk));
        nchunks += nc;
        total += n;
        PairDev& pd = b->host[p];
        pd.nchunks = nc;
        pd.a.partials = b->d_partials + poff;
        poff += (size_t)NMOM * nc;
        // fixed-point units for this shape: a copy of the CTA histogram sees at most
        // ceil(chunk/256)·(256/copies) samples (the single-pair rule, mattes.cu)
        const double per_thread = std::ceil((double)std::min<uint32_t>(n, chunk) / HIST_BLOCK);
        const double lim = 4294967295.0 * 0.98;
        const double coarse_max = std::max(1.0, per_thread * (HIST_BLOCK / copies));
        const double fine_max = std::max(1.0, per_thread * (HIST_BLOCK / fine));
        int k = 22;
        while (k > 0 && std::ldexp(1.0, k) * (2.0 / 3.0) * coarse_max + coarse_max >= lim) --k;
        int kf = FINE_T + 22;
        while (kf > k && (std::ldexp(1.0, kf - FINE_T) * fine_max + fine_max >= lim ||
                          std::ldexp(1.0, kf) * (double)(m->n_samples + 1) >= 0x1p63))
            --kf;
        // the most samples a thread may add with these units (any n or chunk: the pair's own
        // number fits)
        int most = (int)per_thread;
        while (most < (1 << 20) &&
               std::ldexp(1.0, k) * (2.0 / 3.0) * (double)(most + 1) * (HIST_BLOCK / copies) +
                       (double)(most + 1) * (HIST_BLOCK / copies) < lim &&
               std::ldexp(1.0, kf - FINE_T) * (double)(most + 1) * (HIST_BLOCK / fine) +
                       (double)(most + 1) * (HIST_BLOCK / fine) < lim)
            ++most;
        per_thread_max = std::min(per_thread_max, most);
        pd.a.hist_scale = (float)std::ldexp(1.0, k);
        pd.a.fine_scale = (float)std::ldexp(1.0, kf);
        pd.a.fine_shift = kf - k;
        pd.a.hist_inv = std::ldexp(1.0, -kf);
        pd.a.copies = copies;
        pd.a.fine_copies = fine;
    }
    if (poff > b->partials_cap) return set_error(ctx, MI_ERR_INVALID_ARGUMENT, "batch chunk shape too fine");
    b->nchunks = nchunks;
    b->seg_max = (unsigned int)per_thread_max * HIST_BLOCK;
    b->chunk = chunk;
    b->copies = copies;
    b->fine_copies = fine;
    const size_t hs = batch_hist_smem(B, copies, fine), ds = stream_smem(B);
    // raise-only limits: another batch with fewer bins must not lower them under this one
    {
        mi_status ls = raise_smem_limit(ctx, (const void*)k_batch_hist, hs);
        if (ls == MI_OK) ls = raise_smem_limit(ctx, (const void*)k_batch_deriv<true>, ds);
        if (ls == MI_OK) ls = raise_smem_limit(ctx, (const void*)k_batch_deriv<false>, ds);
        if (ls != MI_OK) return ls;
    }
    int occ_h = 0, occ_d = 0;
    MI_CHECK_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_h, k_batch_hist, HIST_BLOCK, hs));
    MI_CHECK_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_d, k_batch_deriv<true>, DERIV_BLOCK, ds));
    b->grid_hist = (int)std::max<int64_t>(1, std::min<int64_t>((total + LEAST_SHARE - 1) / LEAST_SHARE + b->npairs,
                                                               ctx->num_sms * std::max(occ_h, 1)));
    b->grid_deriv = std::max(1, std::min(b->nchunks, ctx->num_sms * std::max(occ_d, 1)));
    if (MI_EXACT_DEFERRED && (size_t)b->grid_hist * b->seg_max > b->exq_len) {
        dev_free(ctx, b->d_exq);
        b->d_exq = nullptr;
        b->exq_len = 0;
        MI_CHECK_CUDA(ctx, dev_alloc(ctx, &b->d_exq, (size_t)b->grid_hist * b->seg_max * sizeof(uint32_t)));
        b->exq_len = (size_t)b->grid_hist * b->seg_max;
    }
    release_graph(b);
    return MI_OK;
}

mi_status upload_pairs(mi_batch* b) {
    std::vector<Work> work(b->npairs);
    for (int p = 0; p < b->npairs; ++p)
        work[p] = Work{((unsigned int)b->metrics[p]->n_samples + UNIT - 1) / UNIT * UNIT, (unsigned int)b->host[p].nchunks};
    MI_CHECK_CUDA(b->ctx, cudaMemcpyAsync(b->d_pairs, b->host.data(), b->host.size() * sizeof(PairDev),
                                          cudaMemcpyHostToDevice, b->ctx->stream));
    MI_CHECK_CUDA(b->ctx, cudaMemcpyAsync(b->d_work, work.data(), work.size() * sizeof(Work), cudaMemcpyHostToDevice,
                                          b->ctx->stream));
    return MI_OK;
}

mi_status launch_pass(mi_batch* b, const mi_rsgd_config& cfg, bool update) {
    cudaStream_t st = b->ctx->stream;
    const int B = b->bins;
    MI_CHECK_CUDA(b->ctx, pdl::launch(k_batch_hist, b->grid_hist, HIST_BLOCK, batch_hist_smem(B, b->copies, b->fine_copies), st,
                                      b->d_pairs, b->d_work, b->npairs, b->seg_max, b->d_exq));
    MI_CHECK_CUDA(b->ctx, pdl::launch(update ? k_batch_deriv<true> : k_batch_deriv<false>, b->grid_deriv, DERIV_BLOCK,
                                      stream_smem(B), st, b->d_pairs, b->d_work, b->npairs, (unsigned int)b->chunk, cfg, b->d_active));
    return MI_OK;
}

// Point maps and optimizer state of every pair at its starting parameters.
mi_status seed_pairs(mi_batch* b, const mi_rsgd_config& cfg, const double* params) {
    for (int p = 0; p < b->npairs; ++p) {
        PairDev& pd = b->host[p];
        mi_metric* m = b->metrics[p];
        const double* pp = params + (size_t)p * b->nparams;
        for (int k = 0; k < b->nparams; ++k) pd.params[k] = pp[k];
        const std::vector<double>& fp = b->fixed_params[p];
        mi_status s = shift_corners(b->kind, pp, b->nparams, fp.empty() ? nullptr : fp.data(), (int)fp.size(), m->fgeo,
                                    pd.corners);
        if (s != MI_OK) return s;
        for (int k = 0; k < b->nparams; ++k) pd.scales[k] = 1.0;
        if (cfg.physical_shift_scales) rsgd::shift_scales(pd.corners, pd.scales);
        rsgd::start(pd.state, cfg, b->nparams);
        AffineForm f;
        s = transform_form(b->kind, pp, b->nparams, fp.empty() ? nullptr : fp.data(), (int)fp.size(), &f);
        if (s != MI_OK) return s;
        pd.P = m->base;
        pd.P.brick_bl = 0;  // the batch walks the sample list by grid index
        if (!point_map_fill(pd.P, f.stage, 1)) return set_error(b->ctx, MI_ERR_INVALID_ARGUMENT, "non-finite point map");
        pd.active = 1;
        pd.evaluations = 0;
        pd.stop_ns = 0ull;
        pd.done = 0u;
        pd.value = 0.0;
        pd.valid = 0.0;
    }
    return upload_pairs(b);
}

// Times each candidate shape on [histogram, derivative] passes at the starting
// point (no optimizer step) and keeps the fastest; cached per (bins, size class).
mi_status autotune(mi_batch* b, const mi_rsgd_config& cfg, const double* params) {
    int64_t total = 0;
    for (mi_metric* m : b->metrics) total += m->n_samples;
    const int cls = (int)std::ceil(std::log2((double)std::max<int64_t>(total, 1)));
    const auto key = std::make_pair(b->bins, cls);
    {
        std::lock_guard<std::mutex> g(g_tune_mu);
        auto it = g_tune.find(key);
        if (it != g_tune.end()) return shape_batch(b, it->second.first, it->second.second);
    }
    const int chunks[] = {2048, 4096, 8192, 16384};
    const int copies_c[] = {2, 4, 8};
    cudaEvent_t e0, e1;
    MI_CHECK_CUDA(b->ctx, cudaEventCreate(&e0));
    MI_CHECK_CUDA(b->ctx, cudaEventCreate(&e1));
    float best = 1e30f;
    int best_chunk = 4096, best_copies = 4;
    mi_status st = MI_OK;
    const size_t coarse_cap = std::max<size_t>(48 * 1024, batch_hist_copies(b->bins, hist_copies(b->bins), 0));
    for (int ch : chunks) {
        for (int cp : copies_c) {
            if (batch_hist_copies(b->bins, cp, 0) > coarse_cap) continue;
            if ((st = shape_batch(b, ch, cp)) != MI_OK) break;
            if ((st = seed_pairs(b, cfg, params)) != MI_OK) break;
            if ((st = launch_pass(b, cfg, false)) != MI_OK) break;  // warm-up
            float acc = 0.0f;
            for (int r = 0; r < 3 && st == MI_OK; ++r) {
                cudaEventRecord(e0, b->ctx->stream);
                st = launch_pass(b, cfg, false);
                cudaEventRecord(e1, b->ctx->stream);
                cudaEventSynchronize(e1);
                float ms = 0.0f;
                cudaEventElapsedTime(&ms, e0, e1);
                acc += ms;
            }
            if (st != MI_OK) break;
            if (acc < best) {
                best = acc;
                best_chunk = ch;
                best_copies = cp;
            }
        }
        if (st != MI_OK) break;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (st != MI_OK) return st;
    {
        std::lock_guard<std::mutex> g(g_tune_mu);
        g_tune[key] = std::make_pair(best_chunk, best_copies);
    }
    return shape_batch(b, best_chunk, best_copies);
}

constexpr int PASSES_PER_GRAPH = 8;

mi_status build_graph(mi_batch* b, const mi_rsgd_config& cfg) {
    release_graph(b);
    cudaStream_t st = b->ctx->stream;
    MI_CHECK_CUDA(b->ctx, cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    mi_status s = MI_OK;
    for (int i = 0; i < PASSES_PER_GRAPH && s == MI_OK; ++i) s = launch_pass(b, cfg, true);
    if (s == MI_OK) {
        cudaError_t e = cudaMemcpyAsync(b->h_active, b->d_active, sizeof(unsigned int), cudaMemcpyDeviceToHost, st);
        if (e != cudaSuccess) s = cuda_status(b->ctx, e, "batch graph");
    }
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(st, &g);
    if (s != MI_OK) {
        if (g) cudaGraphDestroy(g);
        return s;
    }
    if (e != cudaSuccess) return cuda_status(b->ctx, e, "batch graph capture");
    b->graph = g;
    e = cudaGraphInstantiate(&b->exec, g, 0);
    if (e != cudaSuccess) return cuda_status(b->ctx, e, "batch graph instantiate");
    b->graph_passes = PASSES_PER_GRAPH;
    b->graph_cfg = cfg;
    return MI_OK;
}

bool same_cfg(const mi_rsgd_config& a, const mi_rsgd_config& c) {
    return a.iterations == c.iterations && a.minimum_step == c.minimum_step &&
           a.gradient_tolerance == c.gradient_tolerance && a.relaxation == c.relaxation &&
           a.learning_rate == c.learning_rate && a.estimate_learning_rate == c.estimate_learning_rate &&
           a.physical_shift_scales == c.physical_shift_scales;
}

void free_batch(mi_batch* b) {
    if (!b) return;
    cudaSetDevice(b->ctx->device);
    mi_context* ctx = b->ctx;
    cudaStreamSynchronize(ctx->stream);
    release_graph(b);
    dev_free(ctx, b->d_pairs);
    dev_free(ctx, b->d_work);
    dev_free(ctx, b->d_partials);
    dev_free(ctx, b->d_active);
    dev_free(ctx, b->d_marks);
    dev_free(ctx, b->d_exq);
    pinned_free(ctx, b->h_active);
    for (mi_metric* m : b->metrics)
        if (m) mi_metric_destroy(m);
    delete b;
}

}  // namespace
}  // namespace mi

extern "C" {

mi_status mi_batch_create(mi_context* ctx, int npairs, const mi_image* const* fixed, const mi_image* const* moving,
                          const mi_sampling* sampling, int bins, int kind, const double* fixed_params, int nfixed,
                          mi_batch** out) {
    using namespace mi;
    if (!ctx || npairs < 1 || !fixed || !moving || !out) return MI_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    int nparams = 0;
    if (kind == MI_TRANSFORM_AFFINE)
        nparams = 12;
    else if (kind == MI_TRANSFORM_TRANSLATION)
        nparams = 3;
    else
        return set_error(ctx, MI_ERR_INVALID_ARGUMENT, "the batched form takes affine or translation transforms");
    if (kind == MI_TRANSFORM_AFFINE && nfixed != 3) return set_error(ctx, MI_ERR_INVALID_ARGUMENT, "affine needs a centre");
    MI_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    mi_batch* b = new (std::nothrow) mi_batch();
    if (!b) return MI_ERR_OUT_OF_MEMORY;
    b->ctx = ctx;
    b->npairs = npairs;
    b->bins = bins;
    b->kind = kind;
    b->nparams = nparams;
    b->metrics.assign(npairs, nullptr);
    b->fixed_params.resize(npairs);
    b->host.resize(npairs);
    mi_status s = MI_OK;
    size_t max_chunks = 0;
    for (int p = 0; p < npairs && s == MI_OK; ++p) {
        s = mi_metric_create(ctx, fixed[p], moving[p], nullptr, nullptr, sampling ? sampling + p : nullptr, bins,
                             &b->metrics[p]);
        if (s != MI_OK) break;
        mi_metric* m = b->metrics[p];
        if (kind == MI_TRANSFORM_AFFINE) b->fixed_params[p].assign(fixed_params + 3 * p, fixed_params + 3 * p + 3);
        PairDev& pd = b->host[p];
        std::memset(&pd, 0, sizeof(PairDev));
        pd.kind = kind;
        pd.nparams = nparams;
        if (kind == MI_TRANSFORM_AFFINE)
            for (int d = 0; d < 3; ++d) pd.center[d] = fixed_params[3 * p + d];
        // Jacobian form: constant for these families
        AffineForm f;
        std::vector<double> p0(nparams, 0.0);
        if (kind == MI_TRANSFORM_AFFINE) p0[0] = p0[4] = p0[8] = 1.0;
        s = transform_form(kind, p0.data(), nparams, kind == MI_TRANSFORM_AFFINE ? pd.center : nullptr,
                           kind == MI_TRANSFORM_AFFINE ? 3 : 0, &f);
        if (s != MI_OK) break;
        pd.J.nparams = nparams;
        for (int i = 0; i < 3 * nparams; ++i) {
            pd.J.jac0[i] = f.jac0[i];
            for (int e = 0; e < 3; ++e) pd.J.jacc[e][i] = f.jacc[e][i];
        }
        EvalArgs& a = pd.a;
        a.moving = m->moving;
        a.mmask = m->mmask;
        a.samples = m->samples;
        a.fbin = m->fbin;
        a.n = (uint32_t)m->n_samples;
        a.npad = (a.n + 3u) & ~3u;
        a.ghist = m->ws.hist;
        a.gcols = m->ws.hist + (size_t)bins * bins + bins;
        a.reps = 1;
        a.rec_bins = m->ws.rec_bins;
        a.rec_f = m->ws.rec_f;
        a.rec_g = m->ws.rec_g;
        a.vsum = m->ws.vsum;
        a.sync = m->ws.done_counter;
        a.result = m->ws.result;
        max_chunks += (size_t)std::max<int64_t>(1, (m->n_samples + 2047) / 2048);
    }
    if (s == MI_OK) {
        cudaError_t e = dev_alloc(ctx, &b->d_pairs, (size_t)npairs * sizeof(PairDev));
        if (e == cudaSuccess) e = dev_alloc(ctx, &b->d_work, (size_t)2 * npairs * sizeof(Work));
        if (e == cudaSuccess) e = dev_alloc(ctx, &b->d_partials, max_chunks * NMOM * sizeof(double));
        if (e == cudaSuccess) e = dev_alloc(ctx, &b->d_active, sizeof(unsigned int));
        if (e == cudaSuccess) e = pinned_alloc(ctx, reinterpret_cast<void**>(&b->h_active), nullptr);
        if (e == cudaSuccess) e = dev_alloc(ctx, &b->d_marks, 2 * sizeof(unsigned long long));
        if (e != cudaSuccess) s = cuda_status(ctx, e, "mi_batch_create");
        b->partials_cap = max_chunks * NMOM;
    }
    if (s == MI_OK) s = shape_batch(b, 4096, hist_copies(bins));
    if (s != MI_OK) {
        free_batch(b);
        return s;
    }
    *out = b;
    return MI_OK;
}

mi_status mi_batch_destroy(mi_batch* b) {
    if (!b) return MI_ERR_INVALID_ARGUMENT;
    mi::free_batch(b);
    return MI_OK;
}

mi_status mi_batch_register(mi_batch* b, const mi_rsgd_config* cfg, int autotune, double* params_inout,
                            mi_rsgd_result* results) {
    using namespace mi;
    if (!b || !cfg || !params_inout || !results) return MI_ERR_INVALID_ARGUMENT;
    mi_context* ctx = b->ctx;
    MI_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    mi_status s = MI_OK;
    if (autotune && (s = mi::autotune(b, *cfg, params_inout)) != MI_OK) return s;
    if ((s = seed_pairs(b, *cfg, params_inout)) != MI_OK) return s;
    const unsigned int n = (unsigned int)b->npairs;
    MI_CHECK_CUDA(ctx, cudaMemcpyAsync(b->d_active, &n, sizeof(n), cudaMemcpyHostToDevice, ctx->stream));
    if (!b->exec || !same_cfg(b->graph_cfg, *cfg))
        if ((s = build_graph(b, *cfg)) != MI_OK) return s;
    // every pair makes at most iterations + 1 evaluations
    const int max_replays = (cfg->iterations + 1 + b->graph_passes - 1) / b->graph_passes + 1;
    k_stamp<<<1, 1, 0, ctx->stream>>>(b->d_marks);
    for (int r = 0; r < max_replays; ++r) {
        MI_CHECK_CUDA(ctx, cudaGraphLaunch(b->exec, ctx->stream));
        MI_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        if (*b->h_active == 0u) break;
    }
    k_stamp<<<1, 1, 0, ctx->stream>>>(b->d_marks + 1);
    MI_CHECK_CUDA(ctx, cudaGetLastError());
    unsigned long long marks[2] = {0ull, 0ull};
    MI_CHECK_CUDA(ctx, cudaMemcpyAsync(marks, b->d_marks, sizeof(marks), cudaMemcpyDeviceToHost, ctx->stream));
    MI_CHECK_CUDA(ctx, cudaMemcpy(b->host.data(), b->d_pairs, b->host.size() * sizeof(PairDev), cudaMemcpyDeviceToHost));
    b->pair_seconds.assign(b->npairs, 0.0);
    for (int p = 0; p < b->npairs; ++p) {
        const unsigned long long stop = b->host[p].stop_ns ? b->host[p].stop_ns : marks[1];
        b->pair_seconds[p] = stop > marks[0] ? (double)(stop - marks[0]) * 1e-9 : 0.0;
    }
    for (int p = 0; p < b->npairs; ++p) {
        const PairDev& pd = b->host[p];
        for (int k = 0; k < b->nparams; ++k) params_inout[(size_t)p * b->nparams + k] = pd.params[k];
        results[p].value = pd.value;
        results[p].valid = (int64_t)pd.valid;
        results[p].iterations = pd.state.taken;
        results[p].stop_reason = pd.active ? MI_STOP_MAX_ITERATIONS : pd.state.stop;
        results[p].evaluations = pd.evaluations;
    }
    return MI_OK;
}

mi_status mi_batch_pair_seconds(const mi_batch* b, double* seconds, int n) {
    if (!b || !seconds || n < b->npairs) return MI_ERR_INVALID_ARGUMENT;
    if ((int)b->pair_seconds.size() != b->npairs) return MI_ERR_INVALID_ARGUMENT;
    for (int p = 0; p < b->npairs; ++p) seconds[p] = b->pair_seconds[p];
    return MI_OK;
}

mi_status mi_batch_shape(const mi_batch* b, int* chunk, int* copies, int* nchunks) {
    if (!b) return MI_ERR_INVALID_ARGUMENT;
    if (chunk) *chunk = b->chunk;
    if (copies) *copies = b->copies;
    if (nchunks) *nchunks = b->nchunks;
    return MI_OK;
}

}  // extern "C"
