// Multi-resolution pyramid level on the device: recursive (IIR) Gaussian smoothing,
// shrink geometry and linear resampling onto the coarse grid, with the reference's
// arithmetic (registration/method.rs:2416-2580 prepare_level; device counterpart
// cuda/ops/pyramid.rs).
//
//   smoothing   filters/recursive_gaussian.rs:81-290 (axis loop), :472-529 (one line,
//               ITK RecursiveSeparableImageFilter::FilterDataArray), coefficients
//               core/deriche.rs (Deriche / Farnebäck zero-order IIR)
//   shrink      filters/shrink.rs:51-95 (ShrinkImageFilter geometry)
//   resample    transform/resample.rs:226-290 with the linear interpolator
//               (transform/interpolator.rs:29-152)
//
// The volume is smoothed in FP64 from the f32 voxels, axis by axis, and narrowed to
// f32 once at the end, as the reference does. Every FP64 operation is a separately
// rounded __dmul_rn/__dadd_rn/__dsub_rn in the reference's order, so the device
// output is the same bits as a serial FP64 implementation of the same expressions.
#include <cmath>
#include <cstring>
#include <new>
#include <type_traits>
#include <vector>

#include "internal.h"

namespace mi {
void index_to_physical(const mi_geometry& g, double* m);
bool invert3(const double* m, double* inv);
}  // namespace mi

namespace {

// Zero-order Deriche coefficients (core/deriche.rs: Coefficients::new with
// ZeroOrder, the published poles and zero-order column), in the order the line
// recursion reads them: n0..n3, d1..d4, m1..m4, bn1..bn4, bm1..bm4.
struct Deriche {
    double c[20];
};

void deriche_zero_order(double sigmad, Deriche& out) {
    const double w1 = 0.6681, l1 = -1.3932, w2 = 2.0787, l2 = -1.3732;  // poles
    const double a1 = 1.3530, b1 = 1.8151, a2 = -0.3531, b2 = 0.0902;   // zero-order column
    // denominator: compute_d_coefficients
    const double cos1 = std::cos(w1 / sigmad), cos2 = std::cos(w2 / sigmad);
    const double exp1 = std::exp(l1 / sigmad), exp2 = std::exp(l2 / sigmad);
    const double d4 = exp1 * exp1 * exp2 * exp2;
    const double d3 = -2.0 * cos1 * exp1 * exp2 * exp2 - 2.0 * cos2 * exp2 * exp1 * exp1;
    const double d2 = 4.0 * cos2 * cos1 * exp1 * exp2 + exp1 * exp1 + exp2 * exp2;
    const double d1 = -2.0 * (exp2 * cos2 + exp1 * cos1);
    const double sd = 1.0 + d1 + d2 + d3 + d4;
    // numerator: compute_n_coefficients
    const double sin1 = std::sin(w1 / sigmad), sin2 = std::sin(w2 / sigmad);
    double n0 = a1 + a2;
    double n1 = exp2 * (b2 * sin2 - (a2 + 2.0 * a1) * cos2) + exp1 * (b1 * sin1 - (a1 + 2.0 * a2) * cos1);
    double n2 = ((a1 + a2) * cos2 * cos1 - b1 * cos2 * sin1 - b2 * cos1 * sin2) * 2.0 * exp1 * exp2 +
                a2 * exp1 * exp1 + a1 * exp2 * exp2;
    double n3 = exp2 * exp1 * exp1 * (b2 * sin2 - a2 * cos2) + exp1 * exp2 * exp2 * (b1 * sin1 - a1 * cos1);
    const double sn0 = n0 + n1 + n2 + n3;
    // zero order: unit DC gain, symmetric anti-causal part
    const double alpha0 = 2.0 * sn0 / sd - n0;
    n0 = n0 / alpha0;
    n1 = n1 / alpha0;
    n2 = n2 / alpha0;
    n3 = n3 / alpha0;
    const double m1 = n1 - d1 * n0, m2 = n2 - d2 * n0, m3 = n3 - d3 * n0, m4 = -d4 * n0;
    const double sn = n0 + n1 + n2 + n3;
    const double sm = m1 + m2 + m3 + m4;
    const double c[20] = {n0, n1, n2, n3, d1, d2, d3, d4, m1, m2, m3, m4,
                          d1 * sn / sd, d2 * sn / sd, d3 * sn / sd, d4 * sn / sd,
                          d1 * sm / sd, d2 * sm / sd, d3 * sm / sd, d4 * sm / sd};
    std::memcpy(out.c, c, sizeof(c));
}

// a·x + b·y + c·z + d·w, each product rounded and the sum taken left to right
__device__ __forceinline__ double dot4(double a, double x, double b, double y, double c, double z, double d,
                                       double w) {
    return __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(a, x), __dmul_rn(b, y)), __dmul_rn(c, z)), __dmul_rn(d, w));
}

// The line recursion (recursive_gaussian.rs:472-529): a causal and an anti-causal
// fourth-order pass, the border value extended to infinity on both ends, out = causal +
// anti-causal. Both passes have one shape. Walking away from its own border, a pass at
// step j takes a sample x_j, forms
//     v_j = (x_j·c0 + x_{j−1}·c1 + x_{j−2}·c2 + x_{j−3}·c3)
//         − (v_{j−1}·d1 + v_{j−2}·d2 + v_{j−3}·d3 + v_{j−4}·d4)
// (samples before the border are the border value e; a v before the border enters as
// e·b_l instead of v·d_l), and contributes v_j to element j from that end. The causal
// pass takes x_j = element j, the anti-causal one the element before (one nearer its
// border). Every product and sum is separately rounded in the reference's order.
struct Recursion {
    double c0, c1, c2, c3, d1, d2, d3, d4, b1, b2, b3, b4;
    double e, w1, w2, w3, q1, q2, q3, q4;

    __device__ __forceinline__ void start(const Deriche& C, int dir, double border) {
        const double* n = C.c + (dir ? 8 : 0);
        const double* b = C.c + (dir ? 16 : 12);
        c0 = n[0]; c1 = n[1]; c2 = n[2]; c3 = n[3];
        d1 = C.c[4]; d2 = C.c[5]; d3 = C.c[6]; d4 = C.c[7];
        b1 = b[0]; b2 = b[1]; b3 = b[2]; b4 = b[3];
        e = w1 = w2 = w3 = border;
        q1 = q2 = q3 = q4 = 0.0;
    }
    // the sum over the samples, which does not depend on the recursion
    __device__ __forceinline__ double samples(double x) {
        const double a = dot4(x, c0, w1, c1, w2, c2, w3, c3);
        w3 = w2;
        w2 = w1;
        w1 = x;
        return a;
    }
    // BORDER: the step index where it is below 4, else 4
    template <int BORDER = 4>
    __device__ __forceinline__ double next(double a) {
        const double r = dot4(BORDER >= 1 ? q1 : e, BORDER >= 1 ? d1 : b1, BORDER >= 2 ? q2 : e, BORDER >= 2 ? d2 : b2,
                              BORDER >= 3 ? q3 : e, BORDER >= 3 ? d3 : b3, BORDER >= 4 ? q4 : e, BORDER >= 4 ? d4 : b4);
        const double v = __dsub_rn(a, r);
        q4 = q3;
        q3 = q2;
        q2 = q1;
        q1 = v;
        return v;
    }
    template <int BORDER>
    __device__ __forceinline__ double step(double x) {
        return next<BORDER>(samples(x));
    }
};

// A warp takes 16 lines: lanes 0–15 run the causal pass of one line each, lanes 16–31 the
// anti-causal pass of the same lines, both walking at once from opposite ends. Until the
// middle each leaves its v in shared memory; past it each finds the other pass's v there
// and the element is finished. So a line is read twice (the second time from L2) and
// written once, no partial result leaves the chip, and the two serial chains, which are
// what one line costs (five dependent FP64 operations a step), run side by side.
// One-warp CTAs of n·128 B shared memory: seven on an SM at n = 256, where the chain (40
// cycles a step) and the FP64 pipe (15 operations a step, 2 cycles each, 7/4 warps a
// scheduler) are about even. So what stands beside the chain must be little and must not
// join it: steps go in blocks of eight, each block's chain runs beside the next block's
// sample sums, and the shared-memory rows are numbered by step, so that a block's
// accesses are constant offsets from one address. The volume stays FP64 between axes and
// is f32 on both ends: the first pass widens as it reads, the last narrows as it writes.
// 251×256×243: 108 µs for the x axis (y and z, 120 and 113 µs, are k_gauss_segments' now: 106
// and 84 µs); one line per thread with the
// partial results in global memory took 285 µs an axis, and widening and narrowing
// passes of their own another 58 µs.
constexpr int GL = 16;       // lines a warp
constexpr int GB = 8;        // steps a block
constexpr int GROW = 32;     // doubles a shared-memory row: the lanes' v of one step
constexpr int GROW_X = 33;   // in the x-axis pass, which also reads it by columns

// The doubles of shared memory for a line of n: rows for the steps up to its middle.
__host__ __device__ inline size_t gauss_rows(int64_t n) { return (size_t)(n / 2 + 1); }

// Steps j0 … j0 + 7 of both passes (the line's last block may have fewer): a holds the
// block's sample sums and is given the next block's, from its samples xn. A lane's v of
// step j < n/2 is left at its column of row j; past the middle the other pass's v of the
// same element is at the partner lane's column of row n − 1 − j, and done(u, place, out)
// finishes that element.
template <int ROW, class Done>
__device__ __forceinline__ void eight_steps(Recursion& R, int j0, int n, double (&a)[GB], const double (&xn)[GB],
                                            double* part, Done done) {
    const int lane = threadIdx.x, half = n / 2;
    if (j0 > 0 && j0 + GB <= half) {
        double* row = part + j0 * ROW + lane;
#pragma unroll
        for (int u = 0; u < GB; ++u) {
            row[u * ROW] = R.next(a[u]);
            a[u] = R.samples(xn[u]);
        }
    } else if (j0 > half && j0 + GB <= n) {
        double* row = part + (n - 1 - j0) * ROW + (lane ^ GL);
        double o[GB];
#pragma unroll
        for (int u = 0; u < GB; ++u) o[u] = row[-u * ROW];
#pragma unroll
        for (int u = 0; u < GB; ++u) {
            o[u] = __dadd_rn(R.next(a[u]), o[u]);
            a[u] = R.samples(xn[u]);
        }
#pragma unroll
        for (int u = 0; u < GB; ++u) done(u, row - u * ROW, o[u]);
    } else {
        // the line's first block, the one its middle falls in, its last
#pragma unroll
        for (int u = 0; u < GB; ++u) {
            const int j = j0 + u;
            if (j < n) {
                double v;
                if (j0 > 0 || u >= 4)
                    v = R.next(a[u]);
                else
                    v = u == 0 ? R.next<0>(a[u]) : (u == 1 ? R.next<1>(a[u]) : (u == 2 ? R.next<2>(a[u]) : R.next<3>(a[u])));
                if (j < half) {
                    part[j * ROW + lane] = v;
                } else {
                    __syncwarp();  // what the passes left each other is in place
                    // on the middle element of an odd line both passes stand at once
                    double* at = part + (n - 1 - j) * ROW + (lane ^ GL);
                    const double o = __shfl_xor_sync(0xffffffffu, v, GL);
                    done(u, at, __dadd_rn(v, 2 * j + 1 == n ? o : *at));
                }
            }
            a[u] = R.samples(xn[u]);
        }
    }
}

// Axes 1 and 2: lane l of a half walks line 16·CTA + l; neighbouring lines are neighbours in
// memory (128-byte rows of FP64). A lane keeps the samples of two to three blocks
// requested. Lanes past the last line repeat it (and write the same values).
template <typename TI, typename TO>
__global__ void __launch_bounds__(32) k_gauss_strided(const TI* __restrict__ in, TO* __restrict__ out, int64_t nlines,
                                                      int n, int64_t stride, int64_t na, int64_t sb, const Deriche C) {
    extern __shared__ double part[];
    const int dir = threadIdx.x / GL;
    const int64_t L = min((int64_t)blockIdx.x * GL + (threadIdx.x & (GL - 1)), nlines - 1);
    const int64_t first = (L % na) + (L / na) * sb + (dir ? (int64_t)(n - 1) * stride : 0);
    const TI* __restrict__ from = in + first;
    TO* __restrict__ to = out + first;
    const int64_t ds = dir ? -stride : stride;
    // the samples of a block: step j takes element j (causal) or j − 1 (anti-causal) from
    // this lane's end
    auto fetch = [&](int j0, TI (&x)[GB]) {
        if (j0 > 0 && j0 + GB <= n) {
            const TI* p = from + (j0 - dir) * ds;
#pragma unroll
            for (int u = 0; u < GB; ++u) x[u] = p[u * ds];
        } else {
#pragma unroll
            for (int u = 0; u < GB; ++u) x[u] = from[min(max(j0 + u - dir, 0), n - 1) * ds];
        }
    };
    TI ring[2][GB];
    double a[GB], xn[GB];
    fetch(0, ring[0]);
    Recursion R;
    R.start(C, dir, (double)from[0]);
#pragma unroll
    for (int u = 0; u < GB; ++u) a[u] = R.samples((double)ring[0][u]);
    fetch(GB, ring[0]);
    fetch(2 * GB, ring[1]);
    for (int j0 = 0; j0 < n; j0 += 2 * GB) {
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const int j = j0 + b * GB;
            if (j < n) {
#pragma unroll
                for (int u = 0; u < GB; ++u) xn[u] = (double)ring[b][u];
                fetch(j + 3 * GB, ring[b]);
                TO* p = to + j * ds;
                eight_steps<GROW>(R, j, n, a, xn, part, [&](int u, double*, double v) { p[u * ds] = (TO)v; });
            }
        }
    }
}

// Axis 0: a line is contiguous, so the warp moves 32 steps of its 16 lines (from both
// ends) through a shared-memory tile, row by row, requested a tile ahead. Finished
// elements replace what the passes left, and leave line by line at the end.
template <typename TI, typename TO>
__global__ void __launch_bounds__(32) k_gauss_rows(const TI* __restrict__ in, TO* __restrict__ out, int64_t nlines,
                                                   int n, const Deriche C) {
    extern __shared__ double part[];  // the rows, then the tile [32][33]
    constexpr int CH = 32;
    TI* tile = reinterpret_cast<TI*>(part + gauss_rows(n) * GROW_X);
    const int lane = threadIdx.x, dir = lane / GL;
    const int64_t line0 = (int64_t)blockIdx.x * GL;
    const int lines = (int)min((int64_t)GL, nlines - line0);
    const TI* __restrict__ from = in + line0 * n;
    TI f[GL], b[GL];
    auto request = [&](int j0) {
        const int tf = min(j0 + lane, n - 1), tb = n - 1 - min(max(j0 + lane - 1, 0), n - 1);
#pragma unroll
        for (int r = 0; r < GL; ++r) {
            const int row = min(r, lines - 1) * n;
            f[r] = from[row + tf];
            b[r] = from[row + tb];
        }
    };
    auto place = [&]() {
        __syncwarp();  // the last tile has been read
#pragma unroll
        for (int r = 0; r < GL; ++r) {
            tile[r * 33 + lane] = f[r];
            tile[(GL + r) * 33 + lane] = b[r];
        }
        __syncwarp();
    };
    request(0);
    place();
    request(CH);
    Recursion R;
    R.start(C, dir, (double)tile[lane * 33]);
    double a[GB], xn[GB];
#pragma unroll
    for (int u = 0; u < GB; ++u) a[u] = R.samples((double)tile[lane * 33 + u]);
    for (int j0 = 0; j0 < n; j0 += GB) {
        const int next = (j0 + GB) & (CH - 1);  // the next block's place in the tile
        if (next == 0) {
            place();
            request(j0 + GB + CH);
        }
#pragma unroll
        for (int u = 0; u < GB; ++u) xn[u] = (double)tile[lane * 33 + next + u];
        eight_steps<GROW_X>(R, j0, n, a, xn, part, [&](int, double* place, double v) { *place = v; });
    }
    __syncwarp();
    for (int r = 0; r < lines; ++r) {
        TO* row = out + (line0 + r) * n;
#pragma unroll 8
        for (int k = lane; k < n; k += 32)
            row[k] = (TO)(2 * k < n ? part[k * GROW_X + r] : part[(n - 1 - k) * GROW_X + GL + r]);
    }
}

// Axes 1 and 2 of volumes with many lines: a lane walks a whole line, and neither pass leaves
// its results anywhere. The causal pass runs once up to the last segment and keeps its four
// v before every segment of 16; then, segment by segment from the far end, it is run
// again from there into registers and the anti-causal pass follows over the same samples.
// Half as many FP64 operations again as k_gauss_strided (45 an element, whose pipe is 40–50 %
// busy; 22 % there), but 4 doubles of shared memory a line and segment of 16 instead of
// 16, and coefficients from the constant bank: fourteen warps of 32 lines an SM at n = 256
// for seven of 16. Samples are requested a segment ahead, as the steps free the registers
// of the last. n ≥ 20.
constexpr int SEG = 16;
constexpr int SEG_LAST = 20;  // the last segment holds 4 + (n − 4) mod 16 elements, so that the
                              // anti-causal border lies inside it

__host__ __device__ inline int segments(int64_t n) { return (int)((n - 4) / SEG) + 1; }

// A pass's state; its coefficients stay in the constant bank.
struct Walk {
    double w1, w2, w3, q1, q2, q3, q4;
};
// One step (Recursion::step) with coefficients c, denominators d; BORDER below 4: the v before
// the border enter as e·b.
template <int BORDER>
__device__ __forceinline__ double walk(Walk& s, double x, const double* c, const double* d, const double* b, double e) {
    const double a = dot4(x, c[0], s.w1, c[1], s.w2, c[2], s.w3, c[3]);
    const double r = dot4(BORDER >= 1 ? s.q1 : e, BORDER >= 1 ? d[0] : b[0], BORDER >= 2 ? s.q2 : e, BORDER >= 2 ? d[1] : b[1],
                          BORDER >= 3 ? s.q3 : e, BORDER >= 3 ? d[2] : b[2], BORDER >= 4 ? s.q4 : e, BORDER >= 4 ? d[3] : b[3]);
    const double v = __dsub_rn(a, r);
    s.w3 = s.w2;
    s.w2 = s.w1;
    s.w1 = x;
    s.q4 = s.q3;
    s.q3 = s.q2;
    s.q2 = s.q1;
    s.q1 = v;
    return v;
}
// The step at the fixed distance `u` from the border, unrolled.
__device__ __forceinline__ double walk_at(int u, Walk& s, double x, const double* c, const double* d, const double* b,
                                          double e) {
    return u == 0 ? walk<0>(s, x, c, d, b, e)
                  : (u == 1 ? walk<1>(s, x, c, d, b, e)
                            : (u == 2 ? walk<2>(s, x, c, d, b, e)
                                      : (u == 3 ? walk<3>(s, x, c, d, b, e) : walk<4>(s, x, c, d, b, e))));
}

template <typename TI, typename TO>
__global__ void __launch_bounds__(32, 14) k_gauss_segments(const TI* __restrict__ in, TO* __restrict__ out, int64_t nlines,
                                                           int n, int64_t stride, int64_t na, int64_t sb,
                                                           const __grid_constant__ Deriche C) {
    extern __shared__ double kept[];  // the causal v before segment k, row 4(k − 1) + l
    const double *cc = C.c, *cd = C.c + 4, *cb = C.c + 12, *ac = C.c + 8, *ab = C.c + 16;
    const int lane = threadIdx.x;
    const int64_t L = min((int64_t)blockIdx.x * 32 + lane, nlines - 1);
    const int64_t first = (L % na) + (L / na) * sb;
    const TI* __restrict__ from = in + first;
    TO* __restrict__ to = out + first;
    const int nseg = segments(n), last = (nseg - 1) * SEG, count = n - last;  // count in [4, 19]
    const double e = (double)from[0];
    // the causal pass up to the last segment
    Walk f{e, e, e, 0.0, 0.0, 0.0, 0.0};
    {
        // each sample is replaced by the next segment's as it is used
        const TI* p = from;
        const int64_t ahead = SEG * stride;
        TI x[SEG];
#pragma unroll
        for (int u = 0; u < SEG; ++u) x[u] = p[u * stride];
        for (int k = 0; k < nseg - 1; ++k, p += ahead) {
            const bool more = k + 2 < nseg;
            const TI* q = more ? p + ahead : p;
            if (k == 0) {
#pragma unroll
                for (int u = 0; u < 4; ++u) walk_at(u, f, (double)x[u], cc, cd, cb, e);
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) walk<4>(f, (double)x[u], cc, cd, cb, e);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = q[u * stride];
#pragma unroll
            for (int u = 4; u < SEG; ++u) {
                walk<4>(f, (double)x[u], cc, cd, cb, e);
                x[u] = q[u * stride];
            }
            double* row = kept + k * 128 + lane;
            row[0] = f.q1;
            row[32] = f.q2;
            row[64] = f.q3;
            row[96] = f.q4;
        }
    }
    // the next segment's samples and the three before them, requested one by one as the
    // anti-causal steps free the registers of the last ones
    TI x[SEG], w[3];
    auto request = [&](int k, int u) {
        if (k < 0) return;
        const TI* p = from + (int64_t)(k * SEG) * stride;
        x[u] = p[u * stride];
        if (u < 3) w[u] = p[k > 0 ? -(u + 1) * stride : 0];
    };
    const double z = (double)from[(int64_t)(n - 1) * stride];
    Walk g{z, z, z, 0.0, 0.0, 0.0, 0.0};
    double after;  // the sample after the segment
    {
        // the last segment, at the end of SEG_LAST places; f stands before it
        double t[SEG_LAST], v[SEG_LAST];
        const int skip = SEG_LAST - count;
#pragma unroll
        for (int u = 0; u < SEG_LAST; ++u) t[u] = (double)from[(int64_t)max(n - SEG_LAST + u, 0) * stride];
#pragma unroll
        for (int u = 0; u < SEG_LAST; ++u) {
            if (u < skip) continue;
            v[u] = walk<4>(f, t[u], cc, cd, cb, e);
        }
#pragma unroll
        for (int u = SEG_LAST - 1; u >= 0; --u) {
            if (u < skip) continue;
            const double y = walk_at(SEG_LAST - 1 - u, g, u + 1 < SEG_LAST ? t[u + 1 < SEG_LAST ? u + 1 : u] : z, ac, cd, ab, z);
            to[(int64_t)(n - SEG_LAST + u) * stride] = (TO)__dadd_rn(v[u], y);
        }
        after = (double)from[(int64_t)last * stride];
#pragma unroll
        for (int u = 0; u < SEG; ++u) request(nseg - 2, u);
    }
    for (int k = nseg - 2; k >= 0; --k) {
        double t[SEG], v[SEG];
#pragma unroll
        for (int u = 0; u < SEG; ++u) t[u] = (double)x[u];
        if (k > 0) {
            const double* row = kept + (k - 1) * 128 + lane;
            f = Walk{(double)w[0], (double)w[1], (double)w[2], row[0], row[32], row[64], row[96]};
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = walk<4>(f, t[u], cc, cd, cb, e);
        } else {
            f = Walk{e, e, e, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = walk_at(u, f, t[u], cc, cd, cb, e);
        }
#pragma unroll
        for (int u = 4; u < SEG; ++u) v[u] = walk<4>(f, t[u], cc, cd, cb, e);
        TO* p = to + (int64_t)(k * SEG) * stride;
#pragma unroll
        for (int u = SEG - 1; u >= 0; --u) {
            const double y = walk<4>(g, u + 1 < SEG ? t[u + 1 < SEG ? u + 1 : u] : after, ac, cd, ab, z);
            p[u * stride] = (TO)__dadd_rn(v[u], y);
            request(k - 1, SEG - 1 - u);
        }
        after = t[0];
    }
}

// Lines too long for a warp's partial results in shared memory: one line per thread, the
// causal pass left in `mid` (FP64) and read back by the anti-causal one.
template <typename TI, typename TO>
__global__ void k_gauss_long(const TI* __restrict__ in, double* __restrict__ mid, TO* __restrict__ out, int64_t nlines,
                             int64_t n, int64_t stride, int64_t na, int64_t sa, int64_t sb, const Deriche C) {
    for (int64_t L = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; L < nlines; L += (int64_t)gridDim.x * blockDim.x) {
        const int64_t base = (L % na) * sa + (L / na) * sb;
        for (int dir = 0; dir < 2; ++dir) {
            Recursion R;
            const int64_t first = base + (dir ? (n - 1) * stride : 0), ds = dir ? -stride : stride;
            R.start(C, dir, (double)in[first]);
            for (int64_t j = 0; j < n; ++j) {
                const double x = (double)in[first + (j > dir ? j - dir : 0) * ds];
                const double v = j >= 4 ? R.step<4>(x)
                                        : (j == 0 ? R.step<0>(x)
                                                  : (j == 1 ? R.step<1>(x) : (j == 2 ? R.step<2>(x) : R.step<3>(x))));
                const int64_t at = first + j * ds;
                if (!dir)
                    mid[at] = v;
                else
                    out[at] = (TO)__dadd_rn(mid[at], v);
            }
        }
    }
}

// Linear resampling of an f32 volume onto another grid through the identity
// (transform/resample.rs:226-290): output index → physical point (origin-first
// fold), the difference to the input origin, its image under the input's
// physical-to-index matrix (accumulated from 0.0), then the linear interpolator —
// inside iff c ∈ [−0.5, size − 0.5) per axis, corner weights the running products
// of (1 − frac, frac), corners clamped to the buffer, summed in corner order with
// zero-weight corners skipped (interpolator.rs:57-88) — or `fill` outside; narrowed
// to f32.
struct ResampleGeo {
    int64_t isz[3], osz[3];
    double oi2p[9], oorg[3];  // output index → physical
    double ip2i[9], iorg[3];  // input physical → index
};

// LINEAR: the linear interpolator (transform/interpolator.rs:103-152); otherwise the
// nearest-neighbour one (interpolator.rs:36-54: floor(c + 0.5), clamped), both behind
// the same inside test and the same index arithmetic.
template <bool LINEAR>
__global__ void k_resample(const float* __restrict__ in, float* __restrict__ out, ResampleGeo G, double fill) {
    const int64_t n = G.osz[0] * G.osz[1] * G.osz[2];
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        const double idx[3] = {(double)(q % G.osz[0]), (double)((q / G.osz[0]) % G.osz[1]),
                               (double)(q / (G.osz[0] * G.osz[1]))};
        double phys[3], diff[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            double acc = G.oorg[r];
#pragma unroll
            for (int c = 0; c < 3; ++c) acc = __dadd_rn(acc, __dmul_rn(G.oi2p[r * 3 + c], idx[c]));
            phys[r] = acc;
        }
        // the identity AffineTransform's transform_point: mat_vec(I, p) + 0
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            double acc = 0.0;
#pragma unroll
            for (int c = 0; c < 3; ++c) acc = __dadd_rn(acc, __dmul_rn(r == c ? 1.0 : 0.0, phys[c]));
            diff[r] = __dsub_rn(__dadd_rn(acc, 0.0), G.iorg[r]);
        }
        double c[3];
        bool inside = true;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            double acc = 0.0;
#pragma unroll
            for (int j = 0; j < 3; ++j) acc = __dadd_rn(acc, __dmul_rn(G.ip2i[r * 3 + j], diff[j]));
            c[r] = acc;
            inside = inside && c[r] >= -0.5 && c[r] < (double)G.isz[r] - 0.5;
        }
        double v = fill;
        if (inside && !LINEAR) {
            int64_t off = 0, mul = 1;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                int64_t i = (int64_t)floor(__dadd_rn(c[d], 0.5));  // round half up
                i = i < 0 ? 0 : (i > G.isz[d] - 1 ? G.isz[d] - 1 : i);
                off += i * mul;
                mul *= G.isz[d];
            }
            v = (double)__ldg(in + off);
        } else if (inside) {
            double fr[3];
            int64_t b0[3], b1[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double f = floor(c[d]);
                fr[d] = __dsub_rn(c[d], f);
                const int64_t base = (int64_t)f, hi = G.isz[d] - 1;
                b0[d] = base < 0 ? 0 : (base > hi ? hi : base);
                b1[d] = base + 1 < 0 ? 0 : (base + 1 > hi ? hi : base + 1);
            }
            double acc = 0.0;
#pragma unroll
            for (int corner = 0; corner < 8; ++corner) {
                double w = 1.0;
                int64_t off = 0, mul = 1;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const int bit = (corner >> d) & 1;
                    w = __dmul_rn(w, bit ? fr[d] : __dsub_rn(1.0, fr[d]));
                    off += (bit ? b1[d] : b0[d]) * mul;
                    mul *= G.isz[d];
                }
                if (w != 0.0) acc = __dadd_rn(acc, __dmul_rn(w, (double)__ldg(in + off)));
            }
            v = acc;
        }
        out[q] = (float)v;
    }
}

int grid_of(int64_t n, int sms) {
    int64_t g = (n + 255) / 256;
    if (g > (int64_t)sms * 8) g = (int64_t)sms * 8;
    return g < 1 ? 1 : (int)g;
}

size_t gauss_smem(int axis, int64_t n, size_t esize) {
    return gauss_rows(n) * (axis == 0 ? GROW_X : GROW) * 8 + (axis == 0 ? 32 * 33 * esize : 0);
}

// Lines of more than about 1,800 elements do not fit what a CTA may opt in to.
bool long_line(mi_context* ctx, int axis, int64_t n, size_t esize) {
    int optin = 0;
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return gauss_smem(axis, n, esize) > (size_t)optin || n > (1 << 20);
}

// Which of the two strided kernels takes an axis: with `fit` warps of k_gauss_strided on an
// SM and `warps` in all. Its lines' partial results leave room for seven warps or fewer
// from n = 220 on, and with more than two rounds of them k_gauss_segments' half as many
// FP64 operations more cost less than the idle pipe: 83–86 against 62–66 µs at 224³,
// 122–125 against 95 at 256³, 260–265 against 183–191 at 320³, 216 against 113 at
// 512×512×64 (y). With eight warps or two rounds it is the other way round: 37–38 against
// 41–44 µs at 192³, 72 against 91 at 512×512×64 (z), 22 against 40 at 256×256×40 (y).
bool many_lines(int fit, int64_t warps, int sms) { return fit <= 7 && warps > (int64_t)2 * fit * sms; }

// One axis of one volume. `mid`: FP64 scratch for long lines.
template <typename TI, typename TO>
mi_status gauss_axis(mi_context* ctx, const TI* in, double* mid, TO* out, const int64_t* sz, int axis, const Deriche& C) {
    cudaStream_t st = ctx->stream;
    const int64_t n = sz[axis], nlines = sz[0] * sz[1] * sz[2] / n;
    const int64_t stride = axis == 0 ? 1 : (axis == 1 ? sz[0] : sz[0] * sz[1]);
    // line L starts at (L % na)·sa + (L / na)·sb
    const int64_t na = axis == 1 ? sz[0] : nlines, sa = axis == 0 ? n : 1, sb = axis == 1 ? sz[0] * sz[1] : 0;
    const int64_t ctas = (nlines + GL - 1) / GL;
    if (long_line(ctx, axis, n, sizeof(TI)) || ctas > 0x7fffffff) {
        k_gauss_long<TI, TO><<<grid_of(nlines, ctx->num_sms), 256, 0, st>>>(in, mid, out, nlines, n, stride, na, sa, sb, C);
    } else if (axis == 0) {
        if constexpr (std::is_same<TI, float>::value) {  // axis 0 is the first: it reads the image
            const size_t sm = gauss_smem(0, n, sizeof(TI));
            const mi_status s = mi::raise_smem_limit(ctx, (const void*)k_gauss_rows<TI, TO>, sm);
            if (s != MI_OK) return s;
            k_gauss_rows<TI, TO><<<(unsigned)ctas, 32, sm, st>>>(in, out, nlines, (int)n, C);
        }
    } else {
        const size_t sm = gauss_smem(axis, n, sizeof(TI));
        mi_status s = mi::raise_smem_limit(ctx, (const void*)k_gauss_strided<TI, TO>, sm);
        if (s != MI_OK) return s;
        int fit = 0;
        MI_CHECK_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_gauss_strided<TI, TO>, 32, sm));
        if (many_lines(fit, ctas, ctx->num_sms)) {
            const size_t kept = (size_t)(segments(n) - 1) * 4 * 32 * 8;
            s = mi::raise_smem_limit(ctx, (const void*)k_gauss_segments<TI, TO>, kept);
            if (s != MI_OK) return s;
            k_gauss_segments<TI, TO><<<(unsigned)((nlines + 31) / 32), 32, kept, st>>>(in, out, nlines, (int)n, stride, na, sb, C);
            MI_CHECK_CUDA(ctx, cudaGetLastError());
            return MI_OK;
        }
        k_gauss_strided<TI, TO><<<(unsigned)ctas, 32, sm, st>>>(in, out, nlines, (int)n, stride, na, sb, C);
    }
    MI_CHECK_CUDA(ctx, cudaGetLastError());
    return MI_OK;
}

mi_status new_image(mi_context* ctx, const mi_geometry& geo, mi_image** out) {
    const int64_t n = geo.size[0] * geo.size[1] * geo.size[2];
    float* d = nullptr;
    MI_CHECK_CUDA(ctx, mi::image_alloc(ctx, &d, n));
    mi_image* img = new (std::nothrow) mi_image();
    if (!img) {
        mi::dev_free(ctx, d);
        return MI_ERR_OUT_OF_MEMORY;
    }
    img->ctx = ctx;
    img->geo = geo;
    img->data = d;
    img->n = n;
    *out = img;
    return MI_OK;
}

bool geo_valid(const mi_geometry* g) {
    if (!g) return false;
    for (int d = 0; d < 3; ++d)
        if (g->size[d] <= 0 || !(g->spacing[d] > 0.0)) return false;
    return true;
}

}  // namespace

extern "C" {

mi_status mi_image_smooth(mi_context* ctx, const mi_image* in, const double* sigma3, mi_image** out) {
    if (!ctx || !in || !sigma3 || !out) return MI_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    const mi_geometry& g = in->geo;
    for (int d = 0; d < 3; ++d) {
        if (!(sigma3[d] >= 0.0) || !std::isfinite(sigma3[d]))
            return mi::set_error(ctx, MI_ERR_INVALID_ARGUMENT, "smoothing sigma must be finite and >= 0");
        // recursive_gaussian.rs: AxisTooShortForRecursion
        if (sigma3[d] > 0.0 && g.size[d] < 4)
            return mi::set_error(ctx, MI_ERR_INVALID_ARGUMENT,
                                 "axis " + std::to_string(d) + " is shorter than the recursion's 4 samples");
    }
    MI_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    mi_image* res = nullptr;
    mi_status s = new_image(ctx, g, &res);
    if (s != MI_OK) return s;
    const int64_t n = in->n;
    cudaStream_t st = ctx->stream;
    // f32 in, FP64 between axes (two volumes in turn), f32 out
    int axes[3], na = 0;
    bool need_mid = false;
    for (int d = 0; d < 3; ++d)
        if (sigma3[d] > 0.0) {
            axes[na++] = d;
            need_mid = need_mid || long_line(ctx, d, g.size[d], sizeof(double));
        }
    double* v[3] = {nullptr, nullptr, nullptr};  // the two volumes, the long lines' scratch
    cudaError_t e = cudaSuccess;
    if (na > 1) e = mi::dev_alloc(ctx, &v[0], (size_t)n * 8);
    if (e == cudaSuccess && na > 2) e = mi::dev_alloc(ctx, &v[1], (size_t)n * 8);
    if (e == cudaSuccess && need_mid) e = mi::dev_alloc(ctx, &v[2], (size_t)n * 8);
    if (e == cudaSuccess && na == 0) e = cudaMemcpyAsync(res->data, in->data, (size_t)n * 4, cudaMemcpyDeviceToDevice, st);
    for (int i = 0; i < na && e == cudaSuccess && s == MI_OK; ++i) {
        const int d = axes[i];
        Deriche C;
        deriche_zero_order(sigma3[d] / g.spacing[d], C);
        const bool first = i == 0, last = i == na - 1;
        if (first && last)
            s = gauss_axis(ctx, in->data, v[2], res->data, g.size, d, C);
        else if (first)
            s = gauss_axis(ctx, in->data, v[2], v[0], g.size, d, C);
        else if (last)
            s = gauss_axis(ctx, v[(i - 1) & 1], v[2], res->data, g.size, d, C);
        else
            s = gauss_axis(ctx, v[(i - 1) & 1], v[2], v[i & 1], g.size, d, C);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    for (double* p : v) mi::dev_free(ctx, p);
    if (e != cudaSuccess || s != MI_OK) {
        mi_image_free(res);
        return e != cudaSuccess ? mi::cuda_status(ctx, e, "mi_image_smooth") : s;
    }
    *out = res;
    return MI_OK;
}

mi_status mi_shrink_geometry(const mi_geometry* in, const int64_t* factors3, mi_geometry* out) {
    if (!in || !factors3 || !out) return MI_ERR_INVALID_ARGUMENT;
    for (int d = 0; d < 3; ++d)
        if (factors3[d] <= 0 || in->size[d] <= 0) return MI_ERR_INVALID_ARGUMENT;  // InvalidShrinkFactor
    mi_geometry o = *in;
    double delta[3];
    for (int d = 0; d < 3; ++d) {
        const int64_t f = factors3[d];
        o.size[d] = std::max<int64_t>(in->size[d] / f, 1);
        o.spacing[d] = in->spacing[d] * (double)f;
        delta[d] = ((double)in->size[d] - 1.0) / 2.0 - (double)f * ((double)o.size[d] - 1.0) / 2.0;
    }
    // origin + Direction·diag(spacing)·δ, accumulated from 0.0 and added last
    for (int i = 0; i < 3; ++i) {
        double acc = 0.0;
        for (int j = 0; j < 3; ++j) acc += in->direction[i * 3 + j] * in->spacing[j] * delta[j];
        o.origin[i] = in->origin[i] + acc;
    }
    *out = o;
    return MI_OK;
}

static mi_status resample(mi_context* ctx, const mi_image* in, const mi_geometry* grid, double fill, bool linear,
                          mi_image** out) {
    if (!ctx || !in || !grid || !out) return MI_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    if (!geo_valid(grid)) return mi::set_error(ctx, MI_ERR_INVALID_ARGUMENT, "bad output geometry");
    ResampleGeo G;
    double ii2p[9];
    mi::index_to_physical(in->geo, ii2p);
    if (!mi::invert3(ii2p, G.ip2i)) return mi::set_error(ctx, MI_ERR_SINGULAR_DIRECTION, "singular input direction");
    mi::index_to_physical(*grid, G.oi2p);
    for (int d = 0; d < 3; ++d) {
        G.isz[d] = in->geo.size[d];
        G.osz[d] = grid->size[d];
        G.oorg[d] = grid->origin[d];
        G.iorg[d] = in->geo.origin[d];
    }
    MI_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    mi_image* res = nullptr;
    mi_status s = new_image(ctx, *grid, &res);
    if (s != MI_OK) return s;
    const int64_t n = res->n;
    if (linear)
        k_resample<true><<<grid_of(n, ctx->num_sms), 256, 0, ctx->stream>>>(in->data, res->data, G, fill);
    else
        k_resample<false><<<grid_of(n, ctx->num_sms), 256, 0, ctx->stream>>>(in->data, res->data, G, fill);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) {
        mi_image_free(res);
        return mi::cuda_status(ctx, e, linear ? "mi_image_resample" : "mi_image_resample_nearest");
    }
    *out = res;
    return MI_OK;
}

mi_status mi_image_resample(mi_context* ctx, const mi_image* in, const mi_geometry* grid, double fill,
                            mi_image** out) {
    return resample(ctx, in, grid, fill, true, out);
}

mi_status mi_image_resample_nearest(mi_context* ctx, const mi_image* in, const mi_geometry* grid, double fill,
                                    mi_image** out) {
    return resample(ctx, in, grid, fill, false, out);
}

mi_status mi_pyramid_level(mi_context* ctx, const mi_image* fixed, const mi_image* moving, double sigma,
                           int sigma_physical, const int64_t* factors3, mi_image** fixed_level,
                           mi_image** moving_level) {
    if (!ctx || !fixed || !moving || !factors3 || !fixed_level || !moving_level) return MI_ERR_INVALID_ARGUMENT;
    *fixed_level = nullptr;
    *moving_level = nullptr;
    // physical_sigma (method.rs:2344-2350): voxel units scale by the fixed spacing
    double s3[3];
    for (int d = 0; d < 3; ++d) s3[d] = sigma_physical ? sigma : sigma * fixed->geo.spacing[d];
    const bool smooth = s3[0] != 0.0 || s3[1] != 0.0 || s3[2] != 0.0;
    const bool native = factors3[0] == 1 && factors3[1] == 1 && factors3[2] == 1;
    mi_image* sf = nullptr;
    mi_status s = MI_OK;
    if (smooth)
        s = mi_image_smooth(ctx, fixed, s3, &sf);
    else
        s = mi_image_from_device(ctx, fixed->data, &fixed->geo, &sf);
    if (s != MI_OK) return s;
    mi_image* fl = sf;
    if (!native) {
        mi_geometry coarse;
        s = mi_shrink_geometry(&sf->geo, factors3, &coarse);
        if (s == MI_OK) s = mi_image_resample(ctx, sf, &coarse, 0.0, &fl);
        mi_image_free(sf);
        if (s != MI_OK) return s;
    }
    mi_image* ml = nullptr;
    if (smooth)
        s = mi_image_smooth(ctx, moving, s3, &ml);
    else
        s = mi_image_from_device(ctx, moving->data, &moving->geo, &ml);
    if (s != MI_OK) {
        mi_image_free(fl);
        return s;
    }
    *fixed_level = fl;
    *moving_level = ml;
    return MI_OK;
}

}  // extern "C"
