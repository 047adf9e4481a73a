// FP64 sampling of the moving volume, shared by the evaluations that keep every quantity in
// FP64 (moments.cu, bspline.cu): the decisions of a sample from a continuous index that
// is within cerr of the exact chain's, its corners and the linear interpolant.
#pragma once

#include <cstdint>
#include <cstring>

#include "sampler.cuh"

namespace mi {
namespace {

// Thresholds on the upper words of a fraction: nearer than cerr to a cell face, and 1/2 ∓
// 2·cerr. A word equal to the threshold's counts as near it.
struct FracWords {
    int face_lo, face_hi;
    int half_lo, half_hi;
    int easy;  // cerr is small enough for them
};

inline FracWords frac_words(double cerr) {
    auto word = [](double v) {
        long long b;
        std::memcpy(&b, &v, 8);
        return (int)(b >> 32);
    };
    return FracWords{word(cerr), word(1.0 - cerr), word(0.5 - 2.0 * cerr), word(0.5 + 2.0 * cerr), cerr < 0.01 ? 1 : 0};
}

// floor and int conversions by addition: 1.5·2^52 + x has x's integer part in its low word
constexpr double BIG = 6755399441055744.0;
__device__ __forceinline__ double u32_to_f64(uint32_t v) { return __hiloint2double(0x43300000, (int)v) - 4503599627370496.0; }

enum : int { SAMPLE_OFF = 0, SAMPLE_IN = 1, SAMPLE_UNSURE = 2 };

// The inside test, the cell and the fractions of the continuous index c, by integers.
// SAMPLE_UNSURE where the inside test, the mask's rounding or (GRAD) the cell could be
// another at the exact index; SAMPLE_IN does not look at the mask.
template <bool GRAD>
__device__ __forceinline__ int place64(const SamplerParams& P, const FracWords& F, const double* c, int* cell, double* fr) {
    bool inner = true, sure = F.easy != 0;
    int h[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double t = __dadd_rd(c[d], BIG);
        cell[d] = __double2loint(t);
        fr[d] = c[d] - (t - BIG);
        h[d] = __double2hiint(fr[d]);
        inner = inner && __double2hiint(t) == 0x43380000 && (unsigned)cell[d] < (unsigned)(P.msz[d] - 1);
        if (GRAD) sure = sure && h[d] > F.face_lo && h[d] < F.face_hi;
        if (P.has_mmask) sure = sure && (h[d] < F.half_lo || h[d] > F.half_hi);
    }
    if (!inner) {
        // off the interior: c ∈ [−1/2, 0) and [size − 1, size − 1/2) are still inside
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int hi = __double2hiint(__dadd_rd(c[d], BIG)), n = cell[d];
            if (hi != 0x43380000 && hi != 0x4337ffff) {
                sure = false;  // past 32 bits, or not a number
            } else if (n == -1 || n == P.msz[d] - 1) {
                if (F.easy && (n == -1 ? h[d] < F.half_lo : h[d] > F.half_hi)) return SAMPLE_OFF;
                sure = sure && (h[d] < F.half_lo || h[d] > F.half_hi);
            } else if ((unsigned)n >= (unsigned)P.msz[d]) {
                if (F.easy) return SAMPLE_OFF;
            }
        }
    }
    return sure ? SAMPLE_IN : SAMPLE_UNSURE;
}

// Whether the moving mask admits the voxel nearest to an exact continuous index
// (core/coord.rs:185-191: floor(c + 0.5), the sum rounded).
__device__ __forceinline__ bool mask_exact(const SamplerParams& P, const uint8_t* __restrict__ mmask, const double* c) {
    uint32_t at = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double r = floor(__dadd_rn(c[d], 0.5));
        if (!(r >= 0.0 && r < (double)P.msz[d])) return false;
        at += (uint32_t)r * (d == 0 ? 1u : (d == 1 ? P.ms1 : P.ms2));
    }
    return __ldg(mmask + at) != 0;
}

// The same for a sample whose rounding is certain (place64).
__device__ __forceinline__ bool mask64(const SamplerParams& P, const uint8_t* __restrict__ mmask, const int* cell,
                                       const double* fr) {
    uint32_t at = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int r = cell[d] + (__double2hiint(fr[d]) >= 0x3fe00000 ? 1 : 0);
        if ((unsigned)r >= (unsigned)P.msz[d]) return false;
        at += (uint32_t)r * (d == 0 ? 1u : (d == 1 ? P.ms1 : P.ms2));
    }
    return __ldg(mmask + at) != 0;
}

// The cell's corners (order of fetch_corners, each clamped to the volume) by plain loads from
// the x-fastest volume: 3–7 % faster here than eight point fetches of a 3-D texture, on the
// whole grid and on sampled lists, at any rotation, and no array to fill at set-up.
__device__ __forceinline__ void load_corners(const SamplerParams& P, const float* __restrict__ moving, const int* cell,
                                             float* v) {
    uint32_t lo[3], up[3];  // the lower corner's offset, and from it to the upper one's
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const uint32_t step = d == 0 ? 1u : (d == 1 ? P.ms1 : P.ms2);
        lo[d] = (uint32_t)max(cell[d], 0) * step;
        up[d] = (unsigned)cell[d] < (unsigned)(P.msz[d] - 1) ? step : 0u;
    }
    const uint32_t o = lo[0] + lo[1] + lo[2];
#pragma unroll
    for (int t = 0; t < 8; ++t)
        v[t] = __ldg(moving + (o + (t & 1 ? up[0] : 0u) + (t & 2 ? up[1] : 0u) + (t & 4 ? up[2] : 0u)));
}

// transform/interpolator.rs:103-152: the linear interpolant at the fractions of the cell
// with corners v, and its gradient in index space. Infinite (or NaN) wherever a corner is, but
// not always the infinity of the reference's weighted sum: see interpolate_weighted.
template <bool GRAD>
__device__ __forceinline__ double interpolate(const float* v, const double* fr, double* g) {
    const double v0 = v[0], v2 = v[2], v4 = v[4], v6 = v[6];
    const double d00 = (double)v[1] - v0, d10 = (double)v[3] - v2, d01 = (double)v[5] - v4, d11 = (double)v[7] - v6;
    const double x00 = fma(fr[0], d00, v0), x10 = fma(fr[0], d10, v2);
    const double x01 = fma(fr[0], d01, v4), x11 = fma(fr[0], d11, v6);
    const double e0 = x10 - x00, e1 = x11 - x01;
    const double y0 = fma(fr[1], e0, x00), y1 = fma(fr[1], e1, x01);
    const double z = y1 - y0;
    if (GRAD) {
        const double a0 = fma(fr[1], d10 - d00, d00), a1 = fma(fr[1], d11 - d01, d01);
        g[0] = fma(fr[2], a1 - a0, a0);
        g[1] = fma(fr[2], e1 - e0, e0);
        g[2] = z;
    }
    return fma(fr[2], z, y0);
}

// The same as the reference forms it, corner by corner: what the interpolant is where a corner
// is infinite (its differences from the others are NaN above). 130 FP64 operations for 22.
template <bool GRAD>
__device__ __forceinline__ double interpolate_weighted(const float* v, const double* fr, double* g) {
    double val = 0.0, gi[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const double w0 = t & 1 ? fr[0] : 1.0 - fr[0], w1 = t & 2 ? fr[1] : 1.0 - fr[1], w2 = t & 4 ? fr[2] : 1.0 - fr[2];
        const double b = (double)v[t];
        val += w0 * w1 * w2 * b;
        gi[0] += (t & 1 ? 1.0 : -1.0) * (w1 * w2) * b;
        gi[1] += (t & 2 ? 1.0 : -1.0) * (w0 * w2) * b;
        gi[2] += (t & 4 ? 1.0 : -1.0) * (w0 * w1) * b;
    }
    if (GRAD) {
#pragma unroll
        for (int d = 0; d < 3; ++d) g[d] = gi[d];
    }
    return val;
}

}  // namespace
}  // namespace mi
