// Sine and cosine of the normal transform's angles.
#pragma once

namespace rc {

// Sine and cosine of q = 2 pi u rounded to a float, 0 <= u < 1: q less the nearest multiple of pi / 2
// (in three parts, Cody and Waite: at u = 3/4 what is left of q is 1.2e-8, and two parts leave 5.8 ulp
// of error in the cosine; the third takes 8 of a fill's 451 us), then polynomials on [-pi/4, pi/4] fitted as the logarithm's:
// within 1.5 ulp.
__device__ __forceinline__ void sincos_2pi(float u, float* sine, float* cosine) {
    const float q = (2.0f * 3.14159265358979323846f) * u;
    const float biased = __fmaf_rn(u, 4.0f, 12582912.0f), kf = biased - 12582912.0f;
    const int k = __float_as_int(biased);
    const float head = __fmaf_rn(-kf, -0x1.777a5cp-25f, __fmaf_rn(-kf, 0x1.921fb6p+0f, q));
    const float r = __fmaf_rn(-kf, -0x1.ee59dap-50f, head), z = r * r;
    const float ps = __fmaf_rn(__fmaf_rn(-0x1.994386p-13f, z, 0x1.11073ap-7f), z, -0x1.555546p-3f);
    const float pc = __fmaf_rn(__fmaf_rn(0x1.99eb4ap-16f, z, -0x1.6c0c32p-10f), z, 0x1.55554ap-5f);
    const float s = __fmaf_rn(ps * z, r, r), c = __fmaf_rn(z, __fmaf_rn(z, pc, -0.5f), 1.0f);
    const bool odd = k & 1;
    *sine = __int_as_float(__float_as_int(odd ? c : s) ^ ((k << 30) & 0x80000000));
    *cosine = __int_as_float(__float_as_int(odd ? s : c) ^ (((k + 1) << 30) & 0x80000000));
}

}  // namespace rc
