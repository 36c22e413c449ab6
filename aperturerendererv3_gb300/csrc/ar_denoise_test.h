// The denoiser's Welch t-test of one pair of pixels in one channel
// (ComputeTStatisticFinal, core/denoise/denoise.cuh:309-321): T below the
// t-quantile of its degrees of freedom, with
//   w = (t^2 + vB) / max(t^2 + vA + vB, 1e-6),  T = sqrt(0.5 / (1 - w) - 1).
// Host + device.
#pragma once
#include "ar_vec.h"

namespace ar
{
constexpr int kDnQuantiles = 1024;  // T_QUANTILE_LUT_SIZE (core/denoise/t_quantile.cuh:6)

// LookupTQuantile005 (core/denoise/t_quantile.cuh:17-26); the float -> int
// conversion saturates and maps NaN to 0, as the GPU's conversion does.
AR_HD float dn_t_quantile(const float* tq, float nu)
{
    const float f = floorf(nu);
    int i;
    if (f != f) i = 0;
    else if (f >= 2147483648.0f) i = 2147483647;
    else if (f <= -2147483648.0f) i = (-2147483647 - 1);
    else i = (int)f;
    uint32_t idx = (i <= 0) ? 0u : (uint32_t)(i - 1);
    if (idx > kDnQuantiles - 1) idx = kDnQuantiles - 1;
    return tq[idx];
}

// t: the difference of the pixels' theta; vA, vB: their variances of theta; u, lo:
// the sums of their Welch terms.  The reference's operations in its order.
AR_HD bool dn_channel_passes(float t, float vA, float vB, float u, float lo, const float* tq)
{
    const float t2 = t * t;
    const float wAsym = (t2 + vB) / fmaxf(t2 + vA + vB, 1.0e-6f);
    const float T = sqrtf(0.5f / (1.0f - wAsym) - 1.0f);
    const float nu = u * u / lo;
    return T < dn_t_quantile(tq, nu);
}

// The same decision for most pairs from t and the two variances alone.  In exact
// arithmetic 0.5 / (1 - w) = D / (2 vA) with D = t^2 + vA + vB, so with rho = D / vA
// the test passes for 2 <= rho < 2 (1 + q^2) (below 2 the square root's argument
// is negative, T is not a number and the comparison false).  Welch's degrees of
// freedom lie between the smaller of the pixels' own and their sum, so a range
// of pixels bounds q.  DnRho holds the four limits: fails below fail_low,
// passes in [pass_low, pass_high), fails above fail_high, undecided in between
// (dn_channel_passes decides).  1 - w rounds to 2^-22 at most, 2^-22 rho of
// itself; the margins 2^-20 rho + 2^-18 cover that, every other rounding and
// that of 1 / vA.
struct DnRho
{
    float fail_low, pass_low, pass_high, fail_high;
};

// min_f, max_f: the pixels' own degrees of freedom (at least 1)
AR_HD DnRho dn_rho_limits(uint32_t min_f, uint32_t max_f, const float* tq)
{
    // one index further on each side than the rounding of the degrees of freedom can reach
    const uint32_t lo = min_f < 2u ? 0u : min_f - 2u;
    const uint32_t hi = max_f > (uint32_t)kDnQuantiles ? (uint32_t)kDnQuantiles : 2u * max_f;
    const float qh = tq[lo < kDnQuantiles - 1 ? lo : kDnQuantiles - 1], ql = tq[hi < kDnQuantiles - 1 ? hi : kDnQuantiles - 1];
    const float kl = 2.0f * (1.0f + ql * ql), kh = 2.0f * (1.0f + qh * qh);
    DnRho r;
    r.fail_low = 2.0f * (1.0f - 0x1p-17f);
    r.pass_low = 2.0f * (1.0f + 0x1p-17f);
    r.pass_high = kl * (1.0f - (0x1p-18f + 0x1p-20f * kl));
    r.fail_high = kh * (1.0f + (0x1p-18f + 0x1p-20f * kh));
    return r;
}

// Whether a pixel's variance of theta and Welch term are numbers the quick tests
// hold for (equal ones: they differ in how they are rounded); a single pixel for
// which they are not makes its whole tile take dn_channel_passes.
AR_HD bool dn_ordinary(float vth, float up)
{
    return vth == up && (up == 0.0f || (up > 0x1p-50f && up < 0x1p50f));
}

// Pass, fail or (both false) undecided.  A t that is not a number or infinite
// fails; so does a noise-free centre (inv_vA infinite) unless D is in the range
// where the denominator's clamp matters.
AR_HD void dn_channel_quick(float t, float vA, float inv_vA, float vB, const DnRho& r, bool* pass, bool* fail)
{
    const float D = t * t + vA + vB;
    const float rho = D * inv_vA;
    const bool clamped = D <= 2.0e-6f;
    *pass = !clamped && rho >= r.pass_low && rho < r.pass_high;
    *fail = !clamped && !(rho >= r.fail_low && rho <= r.fail_high);
}

// x / y to a few ulp
AR_HD float dn_ratio(float x, float y)
{
#if defined(__CUDA_ARCH__)
    return __fdividef(x, y);
#else
    return x / y;
#endif
}

// The same with the pair's own degrees of freedom nu = (vA + vB)^2 / lo: undecided
// only within the margins of the limits and where nu is within 2^-18 of itself
// of a whole number.  lo: the sum of the Welch terms; k2[i]: 2 (1 + q_i^2).
AR_HD void dn_channel_nu(float t, float vA, float inv_vA, float vB, float lo, const float* k2, bool* pass, bool* fail)
{
    const float D = t * t + vA + vB;
    const float rho = D * inv_vA;
    const float u = vA + vB;
    const float x = fminf(dn_ratio(u * u, lo), 1030.5f);
    // floor(x) by rounding x - 1/2 to an integer
    const float z = x - 0.5f;
    const float fl = (z + 12582912.0f) - 12582912.0f;  // 1.5 2^23
    const bool known = fabsf(z - fl) < 0.5f - fmaf(x, 0x1p-18f, 0x1p-20f) && D > 2.0e-6f && lo > 0x1p-110f;
    int i = (int)fl - 1;
    i = i < 0 ? 0 : (i > kDnQuantiles - 1 ? kDnQuantiles - 1 : i);
    const float k = k2[i];
    const float m = fmaf(k, 0x1p-20f, 0x1p-18f);
    *pass = known && rho >= 2.0f * (1.0f + 0x1p-17f) && rho < k - k * m;
    *fail = known && (rho < 2.0f * (1.0f - 0x1p-17f) || rho > k + k * m);
}
} // namespace ar
