// mph_pairs.cuh - the viscous pair term (e, f) in FP32, shared by the kernels
// of the factored operator.
#pragma once

#include "mph_device.cuh"

namespace mph {

// (e, f) of the pair (i, j) in FP32, as every pair-term kernel evaluates it
// (one function, so that they agree bit for bit): x_j - x_i from the
// two-float positions (the high parts of nearby positions subtract with one
// FP32 rounding at most, so q is within about one FP32 ulp of the FP64
// difference, with no FP64 arithmetic); the exact minimum image only when a
// component is not well inside a quarter of the domain width (a periodic
// image, which also sets *wrap).  e = q / |q|, f = visc mu_ij w'(|q|) / |q|
// within RadiusV, else 0 (main.cpp:2261-2289).
template <int D>
__device__ __forceinline__ void pair_ef(const DevParams& P, int i, int j, int ti, const float* hi, const float* li,
                                        const int* __restrict__ type, const double* __restrict__ pos,
                                        const float* __restrict__ pos32, const float* __restrict__ poslo32,
                                        int* __restrict__ wrap, float* e, float& f)
{
    if (j != i) {
        float hj[3], lj[3];
        int tj;
        if (D == 3) {   // the high part's w holds the type bits (k_permute)
            const float4 h4 = reinterpret_cast<const float4*>(pos32)[j];
            hj[0] = h4.x; hj[1] = h4.y; hj[2] = h4.z;
            tj = __float_as_int(h4.w);
        } else {
            load_f32<D>(pos32, j, hj);
            tj = type[j];
        }
        load_f32<D>(poslo32, j, lj);
        float q32[3] = {0.f, 0.f, 0.f};
        bool inner = true;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            q32[d] = (hj[d] - hi[d]) + (lj[d] - li[d]);
            inner = inner && fabsf(q32[d]) < 0.48f * P.hw32[d];
        }
        if (!inner) {
            *wrap = 1;   // the recomputing inner operator then takes the minimum image
            double xi[3], xj[3], q[3];
            load_vec<D>(pos, i, xi);
            load_vec<D>(pos, j, xj);
            sep_vec<D>(P, xj, xi, q);
#pragma unroll
            for (int d = 0; d < D; ++d) q32[d] = (float)q[d];
        }
        const float r2 = q32[0] * q32[0] + q32[1] * q32[1] + q32[2] * q32[2];
        if (r2 != 0.f && P.rV2_32 - r2 > 0.f) {
            const float inv = rsqrtf(r2);
            const float wd = P.wdA32 * (1.f - (r2 * inv) * P.inv_rv32);
            f = P.vm32[ti][tj] * wd * inv;
#pragma unroll
            for (int d = 0; d < D; ++d) e[d] = q32[d] * inv;
        }
    }
}

}  // namespace mph
