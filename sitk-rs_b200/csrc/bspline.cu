// The Mattes metric through a cubic B-spline free-form deformation: the reference's
// sparse-support path (registration/mattes.rs:722-796 evaluate_sparse_support) with its
// BSplineTransform (transform/bspline.rs), on the metric's own samples, masks, ranges
// and histogram geometry.
//
// The samples are walked in the order of their support cells (sorted once per grid: which
// cell a fixed point lies in is the exact chain's, bs_support). Per sample the fast path
// forms the grid coordinate, the 3 × 4 cubic weights and the displacement in FP64 FMAs,
// the control points already mapped to moving index space, so that the continuous index
// is the affine part plus the displacement; it lies within `cerr` of the reference's, and
// the value within `dv`. Where the inside test, the mask's rounding, the cell, the range or
// the Parzen bin could differ, the sample takes the reference's exact FP64 chain
// (bs_sample): every operation separately rounded in the reference's order — fixed point,
// grid index, valid-region test with its far-limit snap, weights, the displacement
// summed in support order, moving index, mask, inside test, trilinear value. So every
// sample's validity and both Parzen bins are the reference's exactly.
//
//   k_bs_hist   pass 1: the joint histogram (FP64 Parzen taps quantised at the metric's
//               fine unit 2^-kf, added as 16-bit halves to u32 shared-memory copies, which
//               are flushed with u64 atomics) and a record per sample (bins, Parzen fraction, moving gradient) in cell order.
//               Its last CTA forms the tail from the integer histogram (value, and the
//               pRatio·nFactor table into global memory).
//   k_bs_cell_deriv  one or more CTAs per support cell: each valid sample of the cell adds
//               weight_k·∇M[d]·Σ_taps B₃′·pRatio to coefficient (d, support point k) of the
//               cell's 4³·3; a CTA sums its samples and adds each sum once.
//
// Each coefficient receives the sums of the (up to 64) cells that share it through
// FP64 atomics, so the derivative's last bits can differ from run to run; the value,
// the valid count and the histogram are integer-exact and repeat bitwise.
//
// Bound: FP64 operations (about 360 a sample in pass 1, 192 in the derivative, two cycles a
// warp each), the L1's share of the control points and few warps beside the registers that
// takes: pass 1 136 µs (FP64 pipe 33 % busy, L1 60 %) and the derivative 77 µs for 1.68 M
// samples on an 8³ mesh. With the exact chain for every sample (about 1,000 operations,
// twelve of them divisions) and 64-bit shared-memory atomics pass 1 took 341 µs.
#include <cub/device/device_radix_sort.cuh>

#include <cfloat>
#include <cmath>
#include <cstring>
#include <new>

#include "internal.h"
#include "sampler.cuh"
#include "sampler64.cuh"
#include "eval_device.cuh"
#include "point_map.h"

namespace mi {

bool invert3(const double* m, double* inv);

namespace {

constexpr int BS_BLOCK = 256;

// The control-point grid (bspline.rs:209-218) and its valid-region limits, formed on
// the host once per call with the reference's expressions.
struct BSplineDev {
    int64_t gsize[3], gstride[3], nper;
    double gorigin[3], p2i[9];
    double max_limit[3], snap_ulp[3], snap_to[3];
    double gA[9], gb[3];  // fixed grid index → control-grid index (FMA form)
    int zero;             // every coefficient is zero
};

// The bounds of one evaluation's fast path.
struct FastBounds {
    FracWords words;
    double dv;        // on the value
    double inv_bin, dterm;  // reciprocal bin size; on the Parzen term
};

// bspline.rs:94-106, every operation separately rounded in the reference's order
__device__ __forceinline__ double bs_cubic(double u) {
    const double a = fabs(u);
    if (a < 1.0) {
        const double sq = __dmul_rn(a, a);
        return __ddiv_rn(__dadd_rn(__dsub_rn(4.0, __dmul_rn(6.0, sq)), __dmul_rn(__dmul_rn(3.0, sq), a)), 6.0);
    } else if (a < 2.0) {
        const double sq = __dmul_rn(a, a);
        return __ddiv_rn(__dsub_rn(__dadd_rn(__dsub_rn(8.0, __dmul_rn(12.0, a)), __dmul_rn(6.0, sq)), __dmul_rn(sq, a)),
                         6.0);
    }
    return 0.0;
}

// The fixed grid point, origin-seeded (registration/scales.rs:259-271)
__device__ __forceinline__ void fixed_point(const SamplerParams& P, uint32_t i, uint32_t j, uint32_t k, double* x) {
    const double di = (double)i, dj = (double)j, dk = (double)k;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        double acc = P.forigin[r];
        acc = __dadd_rn(acc, __dmul_rn(P.fi2p[r * 3 + 0], di));
        acc = __dadd_rn(acc, __dmul_rn(P.fi2p[r * 3 + 1], dj));
        acc = __dadd_rn(acc, __dmul_rn(P.fi2p[r * 3 + 2], dk));
        x[r] = acc;
    }
}

// The grid index of x (bspline.rs:488-499), the valid-region test with the far-limit
// snap (:504-520) and the support start (:525-557). False outside.
__device__ __forceinline__ bool bs_support(const BSplineDev& S, const double* x, double* idx, int64_t* start) {
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        double acc = -0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) acc = __dadd_rn(acc, __dmul_rn(S.p2i[r * 3 + c], __dsub_rn(x[c], S.gorigin[c])));
        idx[r] = acc;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (fabs(__dsub_rn(idx[d], S.max_limit[d])) <= S.snap_ulp[d])
            idx[d] = S.snap_to[d];
        else if (idx[d] >= S.max_limit[d] || idx[d] < 1.0)
            return false;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) start[d] = (int64_t)floor(__dsub_rn(__dadd_rn(idx[d], 0.5), 1.5));
    return true;
}

// And the 1-D weights.
__device__ __forceinline__ bool bs_locate(const BSplineDev& S, const double* x, double (*w1)[4], int64_t* start) {
    double idx[3];
    if (!bs_support(S, x, idx, start)) return false;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        double u = __dsub_rn(idx[d], (double)start[d]);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            w1[d][t] = bs_cubic(u);
            u = __dsub_rn(u, 1.0);
        }
    }
    return true;
}

enum { BS_OUTSIDE = 0, BS_OUT_OF_RANGE = 1, BS_VALID = 2 };

// One sample through the reference's exact chain: status, and for a
// valid sample the moving Parzen term and bin and the moving physical gradient.
__device__ __noinline__ int bs_sample(const SamplerParams& P, const BSplineDev& S, const double* coef, uint32_t flat,
                         const float* __restrict__ moving, const uint8_t* __restrict__ mmask, double& term, int& mi,
                         double* g) {
    uint32_t i, j, k;
    grid_index(P, flat, i, j, k);
    double x[3], y[3];
    fixed_point(P, i, j, k, x);
    double w1[3][4];
    int64_t start[3];
    // (coefficients that are all zero displace nothing: a registration's first evaluation, whose
    // points all lie on voxels, takes this chain for every sample)
    if (!S.zero && bs_locate(S, x, w1, start)) {
        // bspline.rs:561-585: displacement summed over the 4³ support in order
        // weight q = ((1·wx)·wy)·wz as the reference forms it: the 16 (1·wx)·wy
        // products once, then one product per support point
        double wxy[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) wxy[q] = __dmul_rn(__dmul_rn(1.0, w1[0][q & 3]), w1[1][q >> 2]);
        double disp[3] = {0.0, 0.0, 0.0};
        const int64_t base = start[0] * S.gstride[0] + start[1] * S.gstride[1] + start[2] * S.gstride[2];
#pragma unroll
        for (int tz = 0; tz < 4; ++tz) {
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const double w = __dmul_rn(wxy[q], w1[2][tz]);
                const int64_t cp = base + (q & 3) + (q >> 2) * S.gstride[1] + tz * S.gstride[2];
#pragma unroll
                for (int d = 0; d < 3; ++d) disp[d] = __dadd_rn(disp[d], __dmul_rn(w, coef[d * S.nper + cp]));
            }
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) y[d] = __dadd_rn(x[d], disp[d]);
    } else {
#pragma unroll
        for (int d = 0; d < 3; ++d) y[d] = x[d];
    }
    // the moving continuous index (registration/metric.rs:795-806)
    const double e0 = __dsub_rn(y[0], P.morigin[0]);
    const double e1 = __dsub_rn(y[1], P.morigin[1]);
    const double e2 = __dsub_rn(y[2], P.morigin[2]);
    double c[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        double acc = __dmul_rn(P.mp2i[r * 3 + 0], e0);
        acc = __dadd_rn(acc, __dmul_rn(P.mp2i[r * 3 + 1], e1));
        acc = __dadd_rn(acc, __dmul_rn(P.mp2i[r * 3 + 2], e2));
        c[r] = acc;
    }
    if (P.has_mmask) {
        uint32_t mflat = 0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double r = floor(__dadd_rn(c[d], 0.5));
            if (!(r >= 0.0 && r < (double)P.msz[d])) return BS_OUTSIDE;
            const uint32_t ri = (uint32_t)r;
            mflat += d == 0 ? ri : (d == 1 ? ri * P.ms1 : ri * P.ms2);
        }
        if (!__ldg(mmask + mflat)) return BS_OUTSIDE;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d)
        if (!(c[d] >= -0.5 && c[d] < P.mhi[d])) return BS_OUTSIDE;
    // the value's eight corners serve the gradient too (the same clamped cell)
    float v[8];
    const double mv = exact_value_corners(P, c, moving, v);
    // the interpolant's exact gradient on the same cell, in FP64 (a continuous weight)
    double fl[3], fr[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        fl[d] = floor(c[d]);
        fr[d] = c[d] - fl[d];
    }
    double gi[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const int b0 = t & 1, b1 = (t >> 1) & 1, b2 = t >> 2;
        const double w0 = b0 ? fr[0] : 1.0 - fr[0], wy = b1 ? fr[1] : 1.0 - fr[1], wz = b2 ? fr[2] : 1.0 - fr[2];
        const double b = (double)v[t];
        gi[0] += (b0 ? 1.0 : -1.0) * (wy * wz) * b;
        gi[1] += (b1 ? 1.0 : -1.0) * (w0 * wz) * b;
        gi[2] += (b2 ? 1.0 : -1.0) * (w0 * wy) * b;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) g[d] = gi[0] * P.mp2i[0 * 3 + d] + gi[1] * P.mp2i[1 * 3 + d] + gi[2] * P.mp2i[2 * 3 + d];
    if (mv < P.moving_min || mv > P.moving_max) return BS_OUT_OF_RANGE;
    term = __dsub_rn(__ddiv_rn(mv, P.moving_bin_size), P.moving_nmin);
    mi = parzen_bin(term, P.bins);
    return BS_VALID;
}

// Up to this many coefficients and derivatives cross in a pinned copy, and the host looks for
// the largest coefficient; more are copied from and to the caller's memory, and the device
// looks (one more wait): beyond it the host's copies and its search cost more. 335,000
// samples, the value and with the derivative, µs: 59,049 coefficients 114 and 259 pinned,
// 116 and 325 copied; 89,373: 141 and 375, 130 and 436; 128,625: 176 and 520, 154 and 564;
// 902,289: 917 and 3,158, 502 and 2,852.
constexpr int64_t PINNED_COEFS = 98304;

// The coefficients `from` the host's pinned copy or the device's: kept on the device (`coef`
// where it is not null, for the exact chain), and as control points in moving index space,
// M·coef, one 32-byte row each; the derivative cleared; the largest |coefficient|'s bits (those
// of NaN pass infinity's) into `top` where it is not null.
__global__ void k_bs_points(const SamplerParams P, int64_t nper, const double* __restrict__ from, double* __restrict__ coef,
                            double4* __restrict__ pts, double* __restrict__ deriv, unsigned long long* __restrict__ top) {
    unsigned long long most = 0ull;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nper; q += (int64_t)gridDim.x * blockDim.x) {
        const double x = from[q], y = from[nper + q], z = from[2 * nper + q];
        double4 v;
        v.x = P.mp2i[0] * x + P.mp2i[1] * y + P.mp2i[2] * z;
        v.y = P.mp2i[3] * x + P.mp2i[4] * y + P.mp2i[5] * z;
        v.z = P.mp2i[6] * x + P.mp2i[7] * y + P.mp2i[8] * z;
        v.w = 0.0;
        pts[q] = v;
        if (coef) {
            coef[q] = x;
            coef[nper + q] = y;
            coef[2 * nper + q] = z;
        }
        if (deriv)
            for (int d = 0; d < 3; ++d) deriv[d * nper + q] = 0.0;
        if (top)
            for (double c : {x, y, z}) most = max(most, (unsigned long long)__double_as_longlong(c) & 0x7fffffffffffffffull);
    }
    if (!top) return;
#pragma unroll
    for (int off = 16; off; off >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, off));
    if ((threadIdx.x & 31) == 0 && most) atomicMax(top, most);
}

// The cubic B-spline's four weights at the fraction t ∈ [0, 1] of the support cell.
__device__ __forceinline__ void bs_weights(double t, double* w) {
    const double r = 1.0 - t, t2 = t * t, t3 = t2 * t;
    w[0] = r * r * r * (1.0 / 6.0);
    w[1] = fma(0.5, t3, fma(-1.0, t2, 2.0 / 3.0));
    w[2] = fma(-0.5, t3, fma(0.5, t2, fma(0.5, t, 1.0 / 6.0)));
    w[3] = t3 * (1.0 / 6.0);
}

// The grouping of the samples by support cell (once per grid).
struct CellPlan {
    const uint32_t* order;  // walk position of the j-th sample in cell order
    const uint32_t* cell;   // its cell (ncells: outside)
    const uint32_t* flat;   // its voxel
    const uint8_t* fbin;    // its fixed bin
    const uint32_t* off;    // [cells + 1] first sample of every cell; the rest lie outside
    uint32_t ncells;
};

// The CTA's histogram: a tap of up to 32 bits is added as its lower and upper 16 bits to two
// u32 counters, and the counts to a third part (64-bit shared-memory atomics are
// compare-and-swap loops: with them the atomics took 200 of the pass's 255 µs). A counter
// takes 65,536 samples. In copies, since neighbours in cell order often share a bin pair:
// lane l adds to copy l mod copies; as many as 48 KB hold, the copies four banks apart.
__host__ __device__ inline int bs_copy_words(int B) { return ((2 * B * B + B + 31) & ~31) + 4; }
int bs_copies(int B) {
    int c = 4;
    while (c > 1 && (size_t)c * bs_copy_words(B) * 4 > 48 * 1024) c >>= 1;
    return c;
}
size_t bs_hist_smem(int B) {
    return std::max((size_t)bs_copies(B) * bs_copy_words(B) * 4, ((tail_smem(B) + 15) & ~(size_t)15) + (size_t)B * B * 4);
}

// A sample of pass 1 on its way: the support cell, the fixed grid index, the continuous
// index without and then with the displacement.
struct BsSample {
    uint32_t flat, cell;
    double c[3];
};

// Pass 1: histogram, records (RECORD) and, in the last CTA, the tail. The taps are the cubic
// B-spline of the FP64 fraction f = term − bin (the same polynomial pieces as the affine
// path), rounded to the fine unit 2^-kf of the metric's global histogram. A CTA takes one
// stretch of the cell order, so its lanes read the same control points together; a
// thread takes two neighbours at a time, which share the control points' 1.5 KB (what a
// load returns to 32 lanes, not its one line, is what the L1 has to move: one sample at a
// time took 145 µs for 1.68 M samples on an 8³ mesh, most of it these loads).
constexpr int BS_HIST_BLOCK = 128;

template <bool RECORD>
__global__ void __launch_bounds__(BS_HIST_BLOCK, 3)
k_bs_hist(const __grid_constant__ SamplerParams P, const __grid_constant__ BSplineDev S, const double* __restrict__ coef,
          const double4* __restrict__ pts, const CellPlan C, const FastBounds F, const EvalArgs a, int copies,
          uint32_t per_cta, double fscale, float* __restrict__ pr_out) {
    extern __shared__ __align__(16) unsigned char bsh[];
    unsigned int* bh = reinterpret_cast<unsigned int*>(bsh);
    const int B = P.bins, B2 = B * B, nb = B2 + B, words = bs_copy_words(B);
    for (int q = threadIdx.x; q < copies * words; q += blockDim.x) bh[q] = 0u;
    const uint32_t j0 = blockIdx.x * per_cta, j1 = min(a.n, j0 + per_cta);
    __syncthreads();
    unsigned int* mine = bh + (threadIdx.x & (copies - 1)) * words;
    const uint32_t ncx = (uint32_t)(S.gsize[0] - 3), ncy = (uint32_t)(S.gsize[1] - 3);

    // the affine part of a sample, and its cubic weights in its cell
    auto begin = [&](uint32_t j, BsSample& q, double (&w)[3][4]) {
        const uint32_t cell = __ldg(C.cell + j);
        q.cell = cell;
        q.flat = __ldg(C.flat + j);
        uint32_t i, jj, k;
        grid_index(P, q.flat, i, jj, k);
        const double x[3] = {u32_to_f64(i), u32_to_f64(jj), u32_to_f64(k)};
        const double st[3] = {u32_to_f64(cell % ncx + 1), u32_to_f64(cell / ncx % ncy + 1), u32_to_f64(cell / (ncx * ncy) + 1)};
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            q.c[r] = fma(P.cA[r * 3 + 2], x[2], fma(P.cA[r * 3 + 1], x[1], fma(P.cA[r * 3], x[0], P.cb[r])));
            bs_weights(fma(S.gA[r * 3 + 2], x[2], fma(S.gA[r * 3 + 1], x[1], fma(S.gA[r * 3], x[0], S.gb[r]))) - st[r], w[r]);
        }
    };
    // the decisions, the histogram and the record of the sample at j in cell order
    auto finish = [&](uint32_t j, const BsSample& q) {
        const int fi = __ldg(C.fbin + j);
        int at[3], mi = 0, st;
        double fr[3], g[3], term = 0.0;
        st = place64<true>(P, F.words, q.c, at, fr);
        if (st == SAMPLE_IN && P.has_mmask && !mask64(P, a.mmask, at, fr)) st = SAMPLE_OFF;
        if (st == SAMPLE_IN) {
            float v[8];
            load_corners(P, a.moving, at, v);
            double gi[3];
            const double mv = interpolate<true>(v, fr, gi);
            if (mv < P.moving_min - F.dv || mv > P.moving_max + F.dv) {
                st = SAMPLE_OFF;
            } else {
                term = fma(mv, F.inv_bin, -P.moving_nmin);
                mi = parzen_bin(term - F.dterm, B);
                if (!(mv >= P.moving_min + F.dv && mv <= P.moving_max - F.dv) || mi != parzen_bin(term + F.dterm, B))
                    st = SAMPLE_UNSURE;
                if (RECORD) {
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        g[d] = gi[0] * P.mp2i[0 * 3 + d] + gi[1] * P.mp2i[1 * 3 + d] + gi[2] * P.mp2i[2 * 3 + d];
                }
            }
        }
        if (st == SAMPLE_UNSURE) {
            double te = 0.0, ge[3];
            int me = 0;
            st = bs_sample(P, S, coef, q.flat, a.moving, a.mmask, te, me, ge) == BS_VALID ? SAMPLE_IN : SAMPLE_OFF;
            term = te;
            mi = me;
#pragma unroll
            for (int d = 0; d < 3; ++d) g[d] = ge[d];
        }
        if (st != SAMPLE_IN) {
            if (RECORD) a.rec_bins[j] = 0;
            return;
        }
        const double f = term - (double)mi, h = 1.0 - f, f2 = f * f, f3 = f2 * f;
        const double w[4] = {h * h * h * (1.0 / 6.0), (3.0 * f3 - 6.0 * f2 + 4.0) * (1.0 / 6.0),
                             (-3.0 * f3 + 3.0 * f2 + 3.0 * f + 1.0) * (1.0 / 6.0), f3 * (1.0 / 6.0)};
        unsigned int* row = mine + fi * B + (mi - 1);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const unsigned int tap = __double2uint_rn(w[t] * fscale);
            atomicAdd(row + t, tap & 0xffffu);
            atomicAdd(row + B2 + t, tap >> 16);
        }
        atomicAdd(mine + 2 * B2 + fi, 1u);
        if (RECORD) {
            a.rec_bins[j] = (uint16_t)(mi | (fi << 8));
            a.rec_f[j] = (float)f;
            a.rec_g[j] = (float)g[0];
            a.rec_g[(size_t)a.npad + j] = (float)g[1];
            a.rec_g[2 * (size_t)a.npad + j] = (float)g[2];
        }
    };
    for (uint32_t j = j0 + 2 * threadIdx.x; j < j1; j += 2 * BS_HIST_BLOCK) {
        const bool pair = j + 1 < j1;
        BsSample p, q;
        double wp[3][4], wq[3][4];
        begin(j, p, wp);
        begin(pair ? j + 1 : j, q, wq);
        // both displacements from one cell's control points; neighbours of two cells take a turn
        // each
        const bool same = p.cell == q.cell;
#pragma unroll 1
        for (int turn = 0; turn < (same ? 1 : 2); ++turn) {
            const uint32_t at = turn ? q.cell : p.cell;
            if (at >= C.ncells) continue;
            const uint32_t sx = at % ncx, sy = at / ncx % ncy, sz = at / (ncx * ncy);
            const double4* row = pts + (sx + S.gstride[1] * sy + S.gstride[2] * sz);
            double dp[3] = {0.0, 0.0, 0.0}, dq[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int tz = 0; tz < 4; ++tz) {
                double rp[3] = {0.0, 0.0, 0.0}, rq[3] = {0.0, 0.0, 0.0};
#pragma unroll
                for (int ty = 0; ty < 4; ++ty) {
                    const double4* line = row + tz * S.gstride[2] + ty * S.gstride[1];
                    double sp[3] = {0.0, 0.0, 0.0}, sq[3] = {0.0, 0.0, 0.0};
#pragma unroll
                    for (int tx = 0; tx < 4; ++tx) {
                        const double2 xy = __ldg(reinterpret_cast<const double2*>(line + tx));
                        const double v[3] = {xy.x, xy.y, __ldg(reinterpret_cast<const double*>(line + tx) + 2)};
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            sp[d] = fma(wp[0][tx], v[d], sp[d]);
                            sq[d] = fma(wq[0][tx], v[d], sq[d]);
                        }
                    }
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        rp[d] = fma(wp[1][ty], sp[d], rp[d]);
                        rq[d] = fma(wq[1][ty], sq[d], rq[d]);
                    }
                }
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    dp[d] = fma(wp[2][tz], rp[d], dp[d]);
                    dq[d] = fma(wq[2][tz], rq[d], dq[d]);
                }
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                if (!turn) p.c[d] += dp[d];
                if (same || turn) q.c[d] += dq[d];
            }
        }
        finish(j, p);
        if (pair) finish(j + 1, q);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < nb; q += blockDim.x) {
        unsigned long long v = 0ull;
        for (int e = 0; e < copies; ++e) {
            const unsigned int* part = bh + e * words;
            v += q < B2 ? part[q] + ((unsigned long long)part[B2 + q] << 16) : part[B2 + q];
        }
        if (v) atomicAdd(a.ghist + q, v);
    }
    if (!last_to_arrive(a.sync)) return;
    // the tail once: value slices folded into the result, the pRatio·nFactor table into global
    // memory for the cells, the global histogram re-zeroed
    const TailSmem ts = tail_layout(B, bsh);
    float* pr = reinterpret_cast<float*>(bsh + ((tail_smem(B) + 15) & ~(size_t)15));
    const TailCtx t = tail_prepare(B, P.moving_bin_size, a, ts);
    if (!t.degenerate) {
        if (RECORD) pr_table(B, t, ts, pr);
        value_slices_share(B, a, t, ts, 0, 1);
    } else if (RECORD) {
        for (int q = threadIdx.x; q < B * B; q += blockDim.x) pr[q] = 0.0f;
    }
    __threadfence_block();
    __syncthreads();
    if (RECORD)
        for (int q = threadIdx.x; q < B * B; q += blockDim.x) pr_out[q] = pr[q];
    if (threadIdx.x < 32) fold_value(B, a, t);
    for (int q = threadIdx.x; q < nb; q += blockDim.x) a.ghist[q] = 0ull;
    if (threadIdx.x == 0) a.sync[0] = 0u;
}

// The support cell of every sample, exact, as one index over the (gsize − 3)³ cells, or
// `ncells` outside the transform's valid region. Depends on the fixed points and the grid
// only, so it is formed once per grid.
__global__ void k_bs_cell_of(const SamplerParams P, const BSplineDev S, const uint32_t* __restrict__ samples,
                             uint32_t n, uint32_t ncells, uint32_t* __restrict__ cell, uint32_t* __restrict__ idx) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const uint32_t flat = samples ? __ldg(samples + s) : s;
        uint32_t i, j, k;
        grid_index(P, flat, i, j, k);
        double x[3], at[3];
        int64_t st[3];
        fixed_point(P, i, j, k, x);
        uint32_t c = ncells;
        if (ncells && bs_support(S, x, at, st))
            c = (uint32_t)(st[0] + (S.gsize[0] - 3) * (st[1] + (S.gsize[1] - 3) * st[2]));
        cell[s] = c;
        idx[s] = s;
    }
}

// The rest of the plan from the sorted cells: each cell's first sample (the least position
// whose cell is not below it), and the samples' voxels and fixed bins in cell order.
__global__ void k_bs_plan(const uint32_t* __restrict__ sorted, const uint32_t* __restrict__ order,
                          const uint32_t* __restrict__ samples, const uint8_t* __restrict__ fbin, uint32_t n,
                          uint32_t ncells, uint32_t* __restrict__ off, uint32_t* __restrict__ flat,
                          uint8_t* __restrict__ bin) {
    const uint32_t stride = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t c = t0; c <= ncells; c += stride) {
        uint32_t lo = 0, hi = n;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(sorted + mid) < c)
                lo = mid + 1;
            else
                hi = mid;
        }
        off[c] = lo;
    }
    for (uint32_t j = t0; j < n; j += stride) {
        const uint32_t s = order[j];
        flat[j] = samples ? __ldg(samples + s) : s;
        bin[j] = __ldg(fbin + s);
    }
}

// The records' bins from cell order back to the walk order.
__global__ void k_bs_unsort(const uint32_t* __restrict__ order, const uint16_t* __restrict__ bins, uint32_t n,
                            uint16_t* __restrict__ out) {
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) out[order[j]] = bins[j];
}

// The derivative of a cell's 4³·3 coefficients over a share of the cell's samples (CTA y of
// the cell takes an equal part), summed in the CTA and added once per coefficient. Thread
// t owns the four support points of column (kx, ky) = t mod 16 for the samples
// j ≡ ⌊t/16⌋ (mod 16) of each staged group; the sixteen partial sums are then combined in
// order. The support weights are continuous factors of the derivative, formed in FP32 from
// the FP64 grid index; the sums are FP64. FP32 → FP64 conversions run at an eighth of the
// FP64 pipe's rate, so the gradient is staged in FP64 and the weights are moved into FP64 by
// shifts alone, 2^896 too small (weights are not negative; zeros and subnormal ones keep
// their value); powers of two on the staged gradient and on the sums make up for it, so the
// sums are those of the plain weights. Every sample through 112 conversions on one CTA a
// cell took 102 µs on an 8³ mesh.
constexpr double WEIGHT_UP = 0x1p800, SUM_UP = 0x1p96;  // together 2^896
__device__ __forceinline__ double small_weight(float w) {
    const unsigned int b = __float_as_uint(w);
    return __hiloint2double((int)(b >> 3), (int)(b << 29));
}

__global__ void __launch_bounds__(BS_BLOCK)
k_bs_cell_deriv(const __grid_constant__ SamplerParams P, const __grid_constant__ BSplineDev S, const EvalArgs a,
                const CellPlan C, const float* __restrict__ pr_g, double* __restrict__ deriv) {
    extern __shared__ __align__(16) unsigned char csh[];
    const int B = P.bins;
    double* sg = reinterpret_cast<double*>(csh);         // [BS_BLOCK][4] weighted gradient
    float* sw = reinterpret_cast<float*>(sg + 4 * BS_BLOCK);  // [BS_BLOCK][12] 1-D weights
    float* pr = sw + 12 * BS_BLOCK;                      // B²
    __shared__ double red[3][BS_BLOCK];
    const uint32_t c = blockIdx.x;
    const uint32_t first = C.off[c], count = C.off[c + 1] - first;
    const uint32_t beg = first + (uint32_t)((uint64_t)count * blockIdx.y / gridDim.y);
    const uint32_t end = first + (uint32_t)((uint64_t)count * (blockIdx.y + 1) / gridDim.y);
    if (beg == end) return;
    for (int q = threadIdx.x; q < B * B; q += blockDim.x) pr[q] = __ldg(pr_g + q);
    const int64_t ncx = S.gsize[0] - 3, ncy = S.gsize[1] - 3;
    const int64_t st[3] = {(int64_t)(c % ncx), (int64_t)((c / ncx) % ncy), (int64_t)(c / (ncx * ncy))};
    // thread t: support column (kx, ky) = t & 15 for all four kz, samples j ≡ t >> 4 (mod 16)
    const int t = threadIdx.x, kxy = t & 15, phase = t >> 4;
    const int kx = kxy & 3, ky = kxy >> 2;
    double acc[4][3] = {};
    __syncthreads();
    for (uint32_t base = beg; base < end; base += BS_BLOCK) {
        const uint32_t j = base + t;
        float G[3] = {0.0f, 0.0f, 0.0f}, W[12];
#pragma unroll
        for (int q = 0; q < 12; ++q) W[q] = 0.0f;
        if (j < end) {
            const uint16_t bins = a.rec_bins[j];
            if (bins) {
                const int mi = bins & 0xff, fi = bins >> 8;
                float dw[4];
                bspline3_deriv_taps(a.rec_f[j], dw);
                const float* row = pr + fi * B + (mi - 1);
                const float ws = fmaf(dw[3], row[3], fmaf(dw[2], row[2], fmaf(dw[1], row[1], dw[0] * row[0])));
                G[0] = ws * a.rec_g[j];
                G[1] = ws * a.rec_g[(size_t)a.npad + j];
                G[2] = ws * a.rec_g[2 * (size_t)a.npad + j];
                uint32_t i, jj, kk;
                grid_index(P, __ldg(C.flat + j), i, jj, kk);
                double x[3];
                fixed_point(P, i, jj, kk, x);
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    double g = 0.0;
#pragma unroll
                    for (int q = 0; q < 3; ++q) g += S.p2i[r * 3 + q] * (x[q] - S.gorigin[q]);
                    float u = (float)(g - (double)st[r]);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float au = fabsf(u), sq = au * au;
                        W[r * 4 + q] = au < 1.0f ? (4.0f - 6.0f * sq + 3.0f * sq * au) * (1.0f / 6.0f)
                                                 : (au < 2.0f ? (2.0f - au) * (2.0f - au) * (2.0f - au) * (1.0f / 6.0f)
                                                              : 0.0f);
                        u -= 1.0f;
                    }
                }
            }
        }
        *reinterpret_cast<double2*>(sg + 4 * t) = make_double2((double)G[0] * WEIGHT_UP, (double)G[1] * WEIGHT_UP);
        sg[4 * t + 2] = (double)G[2] * WEIGHT_UP;
#pragma unroll
        for (int q = 0; q < 12; q += 4)
            *reinterpret_cast<float4*>(sw + 12 * t + q) = make_float4(W[q], W[q + 1], W[q + 2], W[q + 3]);
        __syncthreads();
        const int cnt = (int)min((uint32_t)BS_BLOCK, end - base);
#pragma unroll 2
        for (int jj = phase; jj < cnt; jj += 16) {
            const float wxy = sw[12 * jj + kx] * sw[12 * jj + 4 + ky];
            const float4 wz = *reinterpret_cast<const float4*>(sw + 12 * jj + 8);
            const double2 g01 = *reinterpret_cast<const double2*>(sg + 4 * jj);
            const double g2 = sg[4 * jj + 2];
            const double w[4] = {small_weight(wxy * wz.x), small_weight(wxy * wz.y), small_weight(wxy * wz.z),
                                 small_weight(wxy * wz.w)};
#pragma unroll
            for (int kz = 0; kz < 4; ++kz) {
                acc[kz][0] = fma(w[kz], g01.x, acc[kz][0]);
                acc[kz][1] = fma(w[kz], g01.y, acc[kz][1]);
                acc[kz][2] = fma(w[kz], g2, acc[kz][2]);
            }
        }
        __syncthreads();
    }
    // the 16 phases of each column, summed in phase order
    for (int kz = 0; kz < 4; ++kz) {
#pragma unroll
        for (int d = 0; d < 3; ++d) red[d][t] = acc[kz][d] * SUM_UP;
        __syncthreads();
        if (t < 48) {
            const int d = t >> 4, q = t & 15, qx = q & 3, qy = q >> 2;
            const int64_t cp = (st[0] + qx) * S.gstride[0] + (st[1] + qy) * S.gstride[1] + (st[2] + kz) * S.gstride[2];
            double v = 0.0;
#pragma unroll
            for (int ph = 0; ph < 16; ++ph) v += red[d][q + 16 * ph];
            if (v != 0.0) atomicAdd(deriv + d * S.nper + cp, v);
        }
        __syncthreads();
    }
}

}  // namespace

// Host side of the B-spline evaluation (see the entry point below).
mi_status evaluate_bspline(mi_metric* m, const double* fixed18, const double* coef, int64_t ncoef, double* value,
                           double* derivative, int64_t* valid, uint16_t* records = nullptr) {
    mi_context* ctx = m->ctx;
    if (m->metric_kind != MI_METRIC_MATTES)
        return set_error(ctx, MI_ERR_INVALID_ARGUMENT, "the B-spline path is a Mattes-metric evaluation");
    BSplineDev S;
    double mdir[9];
    for (int d = 0; d < 3; ++d) {
        const double sz = fixed18[d];
        S.gsize[d] = sz >= 1.0 ? (int64_t)sz : 0;  // static_cast<SizeValueType>, as ITK truncates
        if (S.gsize[d] == 0) return set_error(ctx, MI_ERR_INVALID_ARGUMENT, "InvalidBSplineDomain: a zero grid size");
        S.gorigin[d] = fixed18[3 + d];
    }
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) mdir[r * 3 + c] = fixed18[9 + r * 3 + c] * fixed18[6 + c];
    if (!invert3(mdir, S.p2i)) return set_error(ctx, MI_ERR_SINGULAR_DIRECTION, "singular B-spline grid direction");
    S.gstride[0] = 1;
    S.gstride[1] = S.gsize[0];
    S.gstride[2] = S.gsize[0] * S.gsize[1];
    S.nper = S.gsize[0] * S.gsize[1] * S.gsize[2];
    if (ncoef != 3 * S.nper)
        return set_error(ctx, MI_ERR_INVALID_ARGUMENT, "coefficient count is not 3 × the control-point count");
    for (int d = 0; d < 3; ++d) {
        // bspline.rs:504-520
        const double max_limit = (double)S.gsize[d] - 0.5 * (3.0 - 1.0) - 1.0;
        const double scale = std::fabs(max_limit) > 1.0 ? std::fabs(max_limit) : 1.0;
        S.max_limit[d] = max_limit;
        S.snap_ulp[d] = 4.0 * DBL_EPSILON * scale;
        S.snap_to[d] = max_limit - 6.0 * DBL_EPSILON * scale;
    }
    MI_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    Workspace& ws = m->ws;
    const bool pinned = ncoef <= PINNED_COEFS;
    if ((size_t)ncoef > m->bs_cap) {
        dev_free(ctx, m->bs_coef);
        dev_free(ctx, m->bs_deriv);
        dev_free(ctx, m->bs_points);
        m->bs_coef = m->bs_deriv = nullptr;
        m->bs_points = nullptr;
        m->bs_cap = 0;
        MI_CHECK_CUDA(ctx, dev_alloc(ctx, &m->bs_coef, (size_t)ncoef * sizeof(double)));
        MI_CHECK_CUDA(ctx, dev_alloc(ctx, &m->bs_deriv, (size_t)ncoef * sizeof(double)));
        MI_CHECK_CUDA(ctx, dev_alloc(ctx, &m->bs_points, (size_t)S.nper * sizeof(double4)));
        m->bs_cap = (size_t)ncoef;
    }
    if (pinned && (size_t)ncoef > m->bs_host_cap) {
        pinned_free(ctx, m->bs_host, m->bs_host_cap * sizeof(double));
        m->bs_host = m->bs_host_dev = nullptr;
        m->bs_host_cap = 0;
        MI_CHECK_CUDA(ctx, pinned_alloc(ctx, (void**)&m->bs_host, (void**)&m->bs_host_dev, (size_t)ncoef * sizeof(double)));
        m->bs_host_cap = (size_t)ncoef;
    }
    // the largest |coefficient|, by its bits
    unsigned long long top = 0ull;
    const auto points = [&](const double* from, double* keep, unsigned long long* most) {
        k_bs_points<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>((S.nper + 127) / 128, (int64_t)ctx->num_sms * 8)), 128,
                      0, st>>>(m->base, S.nper, from, keep, reinterpret_cast<double4*>(m->bs_points),
                               derivative ? m->bs_deriv : nullptr, most);
        return cudaGetLastError();
    };
    if (pinned) {
        std::memcpy(m->bs_host, coef, (size_t)ncoef * sizeof(double));
        // eight at a time
        unsigned long long most[8] = {};
        const auto bits_at = [&](int64_t q) {
            unsigned long long v;
            std::memcpy(&v, coef + q, 8);
            return v & 0x7fffffffffffffffull;
        };
        int64_t q = 0;
        for (; q + 8 <= ncoef; q += 8)
            for (int e = 0; e < 8; ++e) most[e] = std::max(most[e], bits_at(q + e));
        for (; q < ncoef; ++q) most[0] = std::max(most[0], bits_at(q));
        for (unsigned long long v : most) top = std::max(top, v);
        MI_CHECK_CUDA(ctx, points(m->bs_host_dev, m->bs_coef, nullptr));
    } else {
        unsigned long long* most = reinterpret_cast<unsigned long long*>(ws.result);  // (free until the pass)
        MI_CHECK_CUDA(ctx, cudaMemcpyAsync(m->bs_coef, coef, (size_t)ncoef * sizeof(double), cudaMemcpyHostToDevice, st));
        MI_CHECK_CUDA(ctx, cudaMemsetAsync(most, 0, sizeof(*most), st));
        MI_CHECK_CUDA(ctx, points(m->bs_coef, nullptr, most));
        MI_CHECK_CUDA(ctx, cudaMemcpyAsync(ws.host_result, most, sizeof(*most), cudaMemcpyDeviceToHost, st));
        MI_CHECK_CUDA(ctx, cudaStreamSynchronize(st));
        std::memcpy(&top, ws.host_result, sizeof(top));
    }
    const int B = m->bins;
    const uint32_t n = (uint32_t)m->n_samples;
    // The point map without the displacement (the identity stage): c = cA·idx + cb.
    SamplerParams P = m->base;
    const double identity[12] = {1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0};
    if (!point_map_fill(P, identity, 1)) return set_error(ctx, MI_ERR_INVALID_ARGUMENT, "non-finite geometry");
    // The fast path's bounds. Both chains round some 10³ quantities of at most `mag` moving
    // voxels (the affine part's, bounded through P.cerr, and the displacement's) to 2^-53; the
    // grid coordinate's own rounding (of its largest magnitude, `gmag` cells) moves the
    // displacement by at most 4 control-point magnitudes per cell. 2^-40 leaves a factor of
    // 8 over that. A value moves by at most 2·vmax per voxel and axis.
    FastBounds F;
    {
        double cmax = 0.0, gmag = 0.0;
        std::memcpy(&cmax, &top, 8);
        const bool finite = cmax <= DBL_MAX;
        S.zero = cmax == 0.0 ? 1 : 0;
        double to_index = 0.0;
        for (int i = 0; i < 9; ++i) to_index = std::fmax(to_index, std::fabs(P.mp2i[i]));
        for (int r = 0; r < 3; ++r) {
            double fa[3], b = 0.0, mg = 0.0;
            for (int e = 0; e < 3; ++e) {
                fa[e] = 0.0;
                for (int q = 0; q < 3; ++q) fa[e] += S.p2i[r * 3 + q] * P.fi2p[q * 3 + e];
                S.gA[r * 3 + e] = fa[e];
            }
            for (int q = 0; q < 3; ++q) {
                b += S.p2i[r * 3 + q] * (P.forigin[q] - S.gorigin[q]);
                mg += std::fabs(S.p2i[r * 3 + q]) * (std::fabs(P.forigin[q]) + std::fabs(S.gorigin[q]));
                for (int e = 0; e < 3; ++e)
                    mg += std::fabs(S.p2i[r * 3 + q] * P.fi2p[q * 3 + e]) * (double)(m->fgeo.size[e] - 1);
            }
            S.gb[r] = b;
            gmag = std::fmax(gmag, mg);
        }
        const double disp = 3.0 * to_index * cmax;  // of a control point, in moving voxels
        const double cerr = P.cerr + 0x1p-40 * disp * (1.0 + 4.0 * (1.0 + gmag));
        // (coefficients that are not finite, or bounds that mean nothing: the exact chain)
        F.words = frac_words(finite && cerr < 0.01 ? cerr : 0.25);
        if (!finite || !(cerr < 0.01)) F.words.easy = 0;
        F.dv = P.vmax * (8.0 * cerr + 0x1p-48);
        F.inv_bin = P.inv_moving_bin_size;
        F.dterm = F.dv * F.inv_bin + 0x1p-48 * (P.vmax * F.inv_bin + std::fabs(P.moving_nmin) + 1.0);
    }
    EvalArgs a;
    std::memset(&a, 0, sizeof(a));
    a.moving = m->moving;
    a.mmask = m->mmask;
    a.samples = m->samples;
    a.fbin = m->fbin;
    a.n = n;
    a.npad = (n + 3u) & ~3u;
    a.hist_inv = std::ldexp(1.0, -ws.fine_scale_log2);
    a.ghist = ws.hist;
    a.rec_bins = ws.rec_bins;
    a.rec_f = ws.rec_f;
    a.rec_g = ws.rec_g;
    a.vsum = ws.vsum;
    a.sync = ws.done_counter;
    a.result = ws.result;
    a.result_host = ws.host_result_dev;
    const int64_t want = ((int64_t)n + BS_BLOCK - 1) / BS_BLOCK;
    // the samples grouped by support cell: formed once per grid (the cell of a sample
    // depends on the fixed point and the grid only)
    if (!m->bs_have_key || std::memcmp(m->bs_key, fixed18, sizeof(m->bs_key)) != 0) {
        m->bs_have_key = false;
        dev_free(ctx, m->bs_order);
        dev_free(ctx, m->bs_off);
        dev_free(ctx, m->bs_flat);
        dev_free(ctx, m->bs_fbin);
        dev_free(ctx, m->bs_cell);
        m->bs_order = m->bs_off = m->bs_flat = m->bs_cell = nullptr;
        m->bs_fbin = nullptr;
        const bool any = S.gsize[0] > 3 && S.gsize[1] > 3 && S.gsize[2] > 3;
        const int64_t ncells = any ? (S.gsize[0] - 3) * (S.gsize[1] - 3) * (S.gsize[2] - 3) : 0;
        if (ncells >= (int64_t)0x7fffffff)
            return set_error(ctx, MI_ERR_INVALID_ARGUMENT, "B-spline grid too large (≥ 2^31 support cells)");
        m->bs_ncells = ncells;
        const size_t cap = std::max<uint32_t>(n, 1u);
        uint32_t *cell = nullptr, *idx = nullptr;
        void* tmp = nullptr;
        size_t sort_bytes = 0;
        int bits = 1;
        while (bits < 32 && ((int64_t)1 << bits) <= ncells) ++bits;
        const int g = (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)ctx->num_sms * 8));
        cudaError_t e = dev_alloc(ctx, &cell, cap * 4);
        if (e == cudaSuccess) e = dev_alloc(ctx, &idx, cap * 4);
        if (e == cudaSuccess) e = dev_alloc(ctx, &m->bs_cell, cap * 4);
        if (e == cudaSuccess) e = dev_alloc(ctx, &m->bs_order, cap * 4);
        if (e == cudaSuccess) e = dev_alloc(ctx, &m->bs_flat, cap * 4);
        if (e == cudaSuccess) e = dev_alloc(ctx, &m->bs_fbin, cap);
        if (e == cudaSuccess) e = dev_alloc(ctx, &m->bs_off, (size_t)(ncells + 1) * 4);
        if (e == cudaSuccess && n > 0) {
            k_bs_cell_of<<<g, BS_BLOCK, 0, st>>>(P, S, m->samples, n, (uint32_t)ncells, cell, idx);
            e = cudaGetLastError();
            if (e == cudaSuccess)
                e = cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, cell, m->bs_cell, idx, m->bs_order, (int)n, 0, bits, st);
            if (e == cudaSuccess) e = dev_alloc(ctx, &tmp, sort_bytes);
            if (e == cudaSuccess)
                e = cub::DeviceRadixSort::SortPairs(tmp, sort_bytes, cell, m->bs_cell, idx, m->bs_order, (int)n, 0, bits, st);
        }
        if (e == cudaSuccess) {
            k_bs_plan<<<g, BS_BLOCK, 0, st>>>(m->bs_cell, m->bs_order, m->samples, m->fbin, n, (uint32_t)ncells, m->bs_off,
                                              m->bs_flat, m->bs_fbin);
            e = cudaGetLastError();
        }
        dev_free(ctx, tmp);
        dev_free(ctx, cell);
        dev_free(ctx, idx);
        if (e != cudaSuccess) return cuda_status(ctx, e, "B-spline support cells");
        std::memcpy(m->bs_key, fixed18, sizeof(m->bs_key));
        m->bs_have_key = true;
    }
    if (!m->bs_pr) MI_CHECK_CUDA(ctx, dev_alloc(ctx, &m->bs_pr, (size_t)B * B * sizeof(float)));
    const CellPlan C{m->bs_order, m->bs_cell, m->bs_flat, m->bs_fbin, m->bs_off, (uint32_t)m->bs_ncells};
    const size_t hsm = bs_hist_smem(B);
    const size_t csm = (size_t)BS_BLOCK * (4 * sizeof(double) + 12 * sizeof(float)) + (size_t)B * B * sizeof(float);
    const bool rec = derivative || records;
    const void* hist_fn = rec ? (const void*)k_bs_hist<true> : (const void*)k_bs_hist<false>;
    mi_status ls = raise_smem_limit(ctx, hist_fn, hsm);
    if (ls == MI_OK) ls = raise_smem_limit(ctx, (const void*)k_bs_cell_deriv, csm);
    if (ls != MI_OK) return ls;
    // one round of CTAs, each a stretch of whole blocks of sample pairs (more where a counter
    // could otherwise see more than 65,536 samples)
    const int64_t blocks = std::max<int64_t>(1, ((int64_t)n + 2 * BS_HIST_BLOCK - 1) / (2 * BS_HIST_BLOCK));
    int occ = 0;
    MI_CHECK_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, rec ? k_bs_hist<true> : k_bs_hist<false>,
                                                                     BS_HIST_BLOCK, hsm));
    int64_t ctas = std::min<int64_t>(blocks, (int64_t)ctx->num_sms * std::max(occ, 1));
    ctas = std::max<int64_t>(ctas, ((int64_t)n + 60000 * bs_copies(B) - 1) / (60000 * bs_copies(B)));
    const uint32_t per_cta = (uint32_t)((blocks + ctas - 1) / ctas * 2 * BS_HIST_BLOCK);
    const double fscale = std::ldexp(1.0, ws.fine_scale_log2);
    const double4* pts = reinterpret_cast<const double4*>(m->bs_points);
    if (rec)
        k_bs_hist<true><<<(unsigned)ctas, BS_HIST_BLOCK, hsm, st>>>(P, S, m->bs_coef, pts, C, F, a, bs_copies(B), per_cta, fscale,
                                                                m->bs_pr);
    else
        k_bs_hist<false><<<(unsigned)ctas, BS_HIST_BLOCK, hsm, st>>>(P, S, m->bs_coef, pts, C, F, a, bs_copies(B), per_cta, fscale,
                                                                 m->bs_pr);
    if (derivative && m->bs_ncells > 0 && n > 0) {
        // parts of a cell: enough CTAs for about eight on every SM
        const int64_t parts = std::max<int64_t>(1, std::min<int64_t>({(int64_t)ctx->num_sms * 8 / m->bs_ncells,
                                                                      (int64_t)n / m->bs_ncells / BS_BLOCK, 64}));
        k_bs_cell_deriv<<<dim3((unsigned)m->bs_ncells, (unsigned)parts), BS_BLOCK, csm, st>>>(P, S, a, C, m->bs_pr, m->bs_deriv);
    }
    uint16_t* walk_bins = nullptr;
    if (records && n > 0) {
        MI_CHECK_CUDA(ctx, dev_alloc(ctx, &walk_bins, (size_t)n * sizeof(uint16_t)));
        k_bs_unsort<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)ctx->num_sms * 8)), BS_BLOCK, 0, st>>>(
            m->bs_order, ws.rec_bins, n, walk_bins);
    }
    MI_CHECK_CUDA(ctx, cudaGetLastError());
    // (the coefficients have been read before the derivative comes back)
    if (derivative)
        MI_CHECK_CUDA(ctx, cudaMemcpyAsync(pinned ? m->bs_host : derivative, m->bs_deriv, (size_t)ncoef * sizeof(double),
                                           cudaMemcpyDeviceToHost, st));
    if (walk_bins) {
        MI_CHECK_CUDA(ctx, cudaMemcpyAsync(records, walk_bins, (size_t)n * sizeof(uint16_t), cudaMemcpyDeviceToHost, st));
        dev_free(ctx, walk_bins);
    }
    MI_CHECK_CUDA(ctx, cudaStreamSynchronize(st));
    if (derivative && pinned) std::memcpy(derivative, m->bs_host, (size_t)ncoef * sizeof(double));
    if (value) *value = ws.host_result[0];
    if (valid) *valid = (int64_t)ws.host_result[1];
    return MI_OK;
}

}  // namespace mi

extern "C" mi_status mi_metric_value_and_derivative_bspline(mi_metric* m, const double* fixed18, const double* coef,
                                                            int64_t ncoef, double* value, double* derivative,
                                                            int64_t* valid) {
    if (!m || !fixed18 || !coef || !value || ncoef < 1) return MI_ERR_INVALID_ARGUMENT;
    return mi::evaluate_bspline(m, fixed18, coef, ncoef, value, derivative, valid);
}

// Per-sample outcome of the B-spline path in the metric's sample order
// (mi_metric_sample_order): moving bin | fixed bin << 8 for a valid sample, 0
// otherwise. For the exactness tests.
extern "C" mi_status mi_metric_bspline_records(mi_metric* m, const double* fixed18, const double* coef,
                                               int64_t ncoef, uint16_t* records, int64_t n) {
    if (!m || !fixed18 || !coef || !records || ncoef < 1) return MI_ERR_INVALID_ARGUMENT;
    if (n < m->n_samples)
        return mi::set_error(m->ctx, MI_ERR_INVALID_ARGUMENT, "output array shorter than the sample count");
    double v = 0.0;
    return mi::evaluate_bspline(m, fixed18, coef, ncoef, &v, nullptr, nullptr, records);
}
