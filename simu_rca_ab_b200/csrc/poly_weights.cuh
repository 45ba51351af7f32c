// Interpolation weights from the fitted polynomials of weight_poly.h, shared
// by the voxel-blocked SIMT kernel and the tensor-core kernel.
#pragma once

#include "das_common.cuh"
#include "weight_poly.h"

namespace rcabf {

// Weights w[0..TAPS) at fractional offset d in [0, 1), from the degree-DEG
// polynomials.
template <int KIND, int DEG>
__device__ __forceinline__ void poly_weights(float d, float (&w)[KindTraits<KIND>::TAPS])
{
    if constexpr (KIND == K_QUAD3) {
        w[0] = 0.5f * d * (d - 1.0f);
        w[1] = (1.0f - d) * (1.0f + d);
        w[2] = 0.5f * d * (d + 1.0f);
    } else {
        // w_j(u) = E_j(u^2) + u O_j(u^2) and w_{T-1-j}(u) = w_j(-u) = E_j - u O_j:
        // both weights of a mirrored pair from one even and one odd Horner
        // chain in s = u^2 (DEG + 1 FMAs per pair)
        using WP = WeightPoly<KIND, DEG>;
        constexpr int T = KindTraits<KIND>::TAPS;
        static_assert(DEG % 2 == 0, "even degree");
        const float u = fmaf(2.0f, d, -1.0f);
        const float s = u * u;
#pragma unroll
        for (int j = 0; j < WP::HALF; ++j) {
            float e = WP::c(j, DEG);
#pragma unroll
            for (int m = DEG - 2; m >= 0; m -= 2) e = fmaf(e, s, WP::c(j, m));
            float o = WP::c(j, DEG - 1);
#pragma unroll
            for (int m = DEG - 3; m >= 1; m -= 2) o = fmaf(o, s, WP::c(j, m));
            w[j] = fmaf(u, o, e);             // w_j(d)
            w[T - 1 - j] = fmaf(-u, o, e);    // w_{T-1-j}(d) = w_j(1 - d)
        }
    }
}

// The weights of two voxels at once: poly_weights' operations on each half of
// a register pair (fma.rn.f32x2 rounds each half as fmaf does), so the same
// bits for half the instructions.
template <int KIND, int DEG>
__device__ __forceinline__ void poly_weights2(float2 d, float2 (&w)[KindTraits<KIND>::TAPS])
{
    auto both = [](float c) { return make_float2(c, c); };
    if constexpr (KIND == K_QUAD3) {
        const float2 h = __fmul2_rn(both(0.5f), d), one = both(1.0f);
        const float2 dm1 = __fadd2_rn(d, both(-1.0f)), dp1 = __fadd2_rn(d, one);
        w[0] = __fmul2_rn(h, dm1);
        w[1] = __fmul2_rn(make_float2(1.0f - d.x, 1.0f - d.y), dp1);
        w[2] = __fmul2_rn(h, dp1);
    } else {
        using WP = WeightPoly<KIND, DEG>;
        constexpr int T = KindTraits<KIND>::TAPS;
        const float2 u = __ffma2_rn(both(2.0f), d, both(-1.0f));
        const float2 s = __fmul2_rn(u, u), nu = make_float2(-u.x, -u.y);
#pragma unroll
        for (int j = 0; j < WP::HALF; ++j) {
            float2 e = both(WP::c(j, DEG));
#pragma unroll
            for (int m = DEG - 2; m >= 0; m -= 2) e = __ffma2_rn(e, s, both(WP::c(j, m)));
            float2 o = both(WP::c(j, DEG - 1));
#pragma unroll
            for (int m = DEG - 3; m >= 1; m -= 2) o = __ffma2_rn(o, s, both(WP::c(j, m)));
            w[j] = __ffma2_rn(u, o, e);
            w[T - 1 - j] = __ffma2_rn(nu, o, e);
        }
    }
}

}  // namespace rcabf
