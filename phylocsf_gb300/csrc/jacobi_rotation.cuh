// The eigensolver's rotations (k_jacobi, kernels.cu).
#pragma once

namespace pcsf {

// Reciprocal and reciprocal square root of a normal d > 0 (exponent well inside the range) to about
// 2^-44: the leading 24 bits by the FP32 approximation, the rest by one Newton step on two floats,
// put together as integers.  FP64 instructions take 69 clocks each in a chain on this part, FP32 and
// integer ones four.
__device__ __forceinline__ double seed_bits(float y0, float y1, int e)
{
    // (double)y0 + y1 for y0 in [0.5, 1], |y1| < 2^-22, times 2^-e
    const int k = __float_as_int(fmaf(y1, 0x1p44f, 12582912.0f)) - 0x4B400000;             // y1 in units of 2^-44
    return __longlong_as_double(((long long)__float_as_int(y0) << 29) + ((long long)(896 - e) << 52) + ((long long)k << 9));
}
__device__ __forceinline__ double recip_seed(double d)
{
    const long long b = __double_as_longlong(d);
    const float mh = __int_as_float(0x3F800000 | ((int)(b >> 29) & 0x7FFFFF));              // mantissa in [1, 2): 24 bits
    const float ml = (__int_as_float(0x4B000000 | ((int)(b >> 6) & 0x7FFFFF)) - 8388608.0f) * 0x1p-46f;
    float y0;
    asm("rcp.approx.f32 %0, %1;" : "=f"(y0) : "f"(mh));
    const float r = fmaf(-ml, y0, fmaf(-mh, y0, 1.0f));
    return seed_bits(y0, y0 * r, (int)(b >> 52) - 1023);
}
__device__ __forceinline__ double rsqrt_seed(double d)
{
    const long long b = __double_as_longlong(d);
    const int e = (int)(b >> 52) - 1023, odd = e & 1;
    const float mh = __int_as_float((0x3F800000 + (odd << 23)) | ((int)(b >> 29) & 0x7FFFFF));   // [1, 4)
    const float ml = (__int_as_float(0x4B000000 | ((int)(b >> 6) & 0x7FFFFF)) - 8388608.0f) * (odd ? 0x1p-45f : 0x1p-46f);
    float y0;
    asm("rsqrt.approx.f32 %0, %1;" : "=f"(y0) : "f"(mh));
    const float p = y0 * y0, pl = fmaf(y0, y0, -p);
    const float r = fmaf(-ml, p, fmaf(-mh, pl, fmaf(-mh, p, 1.0f)));
    return seed_bits(y0, 0.5f * y0 * r, (e - odd) / 2);
}

// 1 / d and sqrt(x), rounded to nearest, of normal d, x > 0 with their seeds y: one residual correction,
// off by ~2^-36 of the last place before its rounding.  That does not tell the side of a tie where the
// operand lies few last places from a power of two or four, as 1 + theta^2 does for every theta below
// 2^-21.  There the value is known: 1 / (1 - k 2^-53) = 1 + k 2^-53 + k^2 2^-106, for odd k just above the
// tie, and half of k, rounded up, in the bits of the result (b: the operand's, less those of 1.0).
// sqrt(1 + k 2^-52) = 1 + k 2^-53 - k^2 2^-107 and sqrt(1 - k 2^-53) = 1 - k 2^-54 - k^2 2^-109 lie for odd k
// just below the tie, so that they round as the root of the operand with its last bit cleared, whose own
// value is next to a double: settle_root clears it.  (After the correction, the same choice between two
// results lengthened a round of the eigensolver by about 60 clocks instead of 25.)
constexpr long long ONE_BITS = 1023ll << 52, NEAR_BITS = 1ll << 20;
__device__ __forceinline__ double recip_rn(double d, double y)
{
    const long long b = __double_as_longlong(d) - ONE_BITS, k = -b & ((1ll << 52) - 1);    // places below a power of two
    const double v = __fma_rn(y, __fma_rn(-d, y, 1.0), y);
    return k < NEAR_BITS ? __longlong_as_double(ONE_BITS - (b + k) + ((k + 1) >> 1)) : v;
}
__device__ __forceinline__ double settle_root(double x)
{
    // the exponent's lowest bit, as an even power's, and the 31 bits after it all zeros or all ones
    const int hi = __double2hiint(x), lo = __double2loint(x);
    const bool near = __funnelshift_l(lo, hi - (int)(ONE_BITS >> 32), 11) + 1u <= 1u;
    return __hiloint2double(hi, near ? lo & ~1 : lo);
}
__device__ __forceinline__ double sqrt_rn(double x, double y)
{
    const double g = x * y;
    return __fma_rn(__fma_rn(-g, g, x), 0.5 * y, g);
}

// The rotation (c, s) that annihilates apq != 0: theta = (aqq - app) / (2 apq), t = sign(theta) /
// (|theta| + sqrt(theta^2 + 1)), c = 1 / sqrt(t^2 + 1), s = t c, each operation rounded to nearest.
// Quotients and roots are seeds (above) with one residual correction in FP64 (Markstein, IBM J. Res.
// Dev. 34 (1990) 111): an error of ~2^-88 before the final rounding, so that, with the ties that
// recip_rn and settle_root settle, they round as the library's do (it would take about 2^35 operations to
// meet one that does not), in 5 x 69 + 90 clocks for a root and its reciprocal instead of 705 + 459
// (the ties cost the omega test of six alignments 1 %).  Operands far from 1, a theta that may overflow
// (its correction would make a NaN of it) and |theta| beyond 2^300 take the library's operations.
__device__ __forceinline__ void jac_rotation(double app, double aqq, double apq, double &c, double &s)
{
    const double num = aqq - app, den = 2.0 * apq, ad = fabs(den);
    const int en = (__double2hiint(num) >> 20) & 0x7FF, ed = __double2hiint(ad) >> 20;
    double theta;
    if ((num == 0.0 || (en > 223 && en < 1823)) && ed > 223 && ed < 1823 && en - ed < 1000) {
        const double y = recip_seed(ad), q = num * y;
        theta = __fma_rn(__fma_rn(-q, ad, num), y, q);
        if (den < 0.0) theta = -theta;
    } else {
        theta = num / den;
    }
    double t;
    if (fabs(theta) < 0x1p300) {
        const double x = settle_root(__fma_rn(theta, theta, 1.0));
        const double d = fabs(theta) + sqrt_rn(x, rsqrt_seed(x));
        t = recip_rn(d, recip_seed(d));
        if (!(theta >= 0.0)) t = -t;
    } else {
        t = (fabs(theta) > 1e150) ? 0.5 / theta
            : (theta >= 0.0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(__fma_rn(theta, theta, 1.0)));
    }
    const double u = settle_root(__fma_rn(t, t, 1.0));      // in [1, 2]
    const double y = rsqrt_seed(u), v = sqrt_rn(u, y);
    c = __fma_rn(y, __fma_rn(-v, y, 1.0), y);
    s = t * c;
}

}  // namespace pcsf
