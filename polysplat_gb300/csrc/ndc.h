// Pixel coordinate of a normalised device coordinate,
//     float(((v + 1.0) * S - 1.0) * 0.5)   in double (preprocess.cu:78-81),
// bit for bit in float arithmetic for the values that matter.
//
// The double form costs three FP64 operations and two conversions per
// coordinate, and FP64 runs at 2 lanes per clock and SM here against 128 for
// FP32: a frame of 20 M Gaussians at 7680x4320 went from 5074 to 5017 us with
// the float form (at 3 M Gaussians the FP64 pipe hides behind the kernel's
// other work: 875 us either way).  For
// 2^-10 <= |v| < 2^20 and S <= 2^14 every step of the double form is exact
// (at most 48 bits), so its result is the exact (v S + S - 1) / 2 rounded
// once.  Here v S = p + e exactly (fused multiply-add), p + (S - 1) = s + t
// exactly (Knuth's two-sum), and t and e are multiples of ulp(v) whose sum
// needs at most 24 bits, so s + (t + e) rounds once as well.  Other values
// (within 2^-10 of the image centre, far outside, infinite, NaN) take the
// double form.
#pragma once

#ifdef __CUDACC__
#define GSR_NDC_FN __device__ __forceinline__
#define GSR_NDC_MUL(a, b) __fmul_rn(a, b)
#define GSR_NDC_ADD(a, b) __fadd_rn(a, b)
#define GSR_NDC_SUB(a, b) __fsub_rn(a, b)
#define GSR_NDC_FMA(a, b, c) __fmaf_rn(a, b, c)
#define GSR_NDC_ABS(a) fabsf(a)
#else  // host check: built with -ffp-contract=off
#include <cmath>
#define GSR_NDC_FN inline
#define GSR_NDC_MUL(a, b) ((a) * (b))
#define GSR_NDC_ADD(a, b) ((a) + (b))
#define GSR_NDC_SUB(a, b) ((a) - (b))
#define GSR_NDC_FMA(a, b, c) std::fma(a, b, c)
#define GSR_NDC_ABS(a) std::fabs(a)
#endif

namespace gsr_ndc {

GSR_NDC_FN float to_pix_double(float v, int S) { return (float)(((v + 1.0) * S - 1.0) * 0.5); }

GSR_NDC_FN float to_pix(float v, int S)
{
    const float a = GSR_NDC_ABS(v);
    if (!(a >= 0.0009765625f && a < 1048576.0f && S <= 16384)) return to_pix_double(v, S);
    const float n = (float)S, c = n - 1.0f;
    const float p = GSR_NDC_MUL(v, n);
    const float e = GSR_NDC_FMA(v, n, -p);
    const float s = GSR_NDC_ADD(p, c);
    const float b = GSR_NDC_SUB(s, p);
    const float t = GSR_NDC_ADD(GSR_NDC_SUB(p, GSR_NDC_SUB(s, b)), GSR_NDC_SUB(c, b));
    return 0.5f * GSR_NDC_ADD(s, GSR_NDC_ADD(t, e));
}

}  // namespace gsr_ndc
