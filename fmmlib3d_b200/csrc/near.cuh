// Elementary functions of the FP64 near-field pair loops: fast paths for
// ordinary arguments, with a flag for the others.  A warp tests the flag once
// for all its pairs and repeats them with the library functions if it is set.
#pragma once

namespace fmm {

// Exponent words of the range in which rsqrt_near needs no care: 2^-975 .. 2^961.
constexpr unsigned kRsqrtLow = 0x03000000u, kRsqrtSpan = 0x79000000u;

// 1/sqrt(x): the hardware's approximation (relative error below 2^-19) and one step
// of Halley's iteration, y (1 + e/2 + 3 e^2/8) with e = 1 - x y^2, which cubes the
// error.  Zeros, infinities, NaN and numbers near the ends of the range need the
// library function: `odd` collects the largest distance of x's exponent word from
// the start of the ordinary range; with LIB such a number takes the library function.
template <bool LIB>
__device__ __forceinline__ double rsqrt_near(double x, unsigned &odd)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    y = fma(y * e, fma(e, 0.375, 0.5), y);
    const unsigned at = (unsigned)__double2hiint(x) - kRsqrtLow;
    if (LIB) {
        if (at > kRsqrtSpan) y = rsqrt(x);
    } else {
        odd = max(odd, at);
    }
    return y;
}

// sin and cos of x for |x| < 2^17: x - n pi/2 with pi/2 as the sum of two doubles
// (Cody and Waite; the products n c exact in the fused multiply-add, the sum's
// error below n 2^-107), then the Taylor series to degree 15 and 16 on |y| <= pi/4
// (remainders 5e-17 and 2e-18).  Larger arguments need the library function: `odd`
// collects the largest exponent word.
constexpr unsigned kSinCosMax = 0x41000000u;   // exponent word of 2^17
template <bool LIB>
__device__ __forceinline__ void sincos_near(double x, double &s, double &c, unsigned &odd)
{
    const double shift = 6755399441055744.0;   // 1.5 2^52: adding it rounds to an integer in the low word
    const double t = fma(x, 0.63661977236758134308, shift);
    const int n = __double2loint(t);
    const double nd = t - shift;
    double y = fma(-nd, 1.5707963267948965580, x);       // pi/2 rounded
    y = fma(-nd, 6.1232339957367660359e-17, y);          // and the rest
    const double z = y * y;
    double a = fma(z, -1.0 / 1307674368000.0, 1.0 / 6227020800.0);
    double b = fma(z, 1.0 / 20922789888000.0, -1.0 / 87178291200.0);
    a = fma(z, a, -1.0 / 39916800.0);
    b = fma(z, b, 1.0 / 479001600.0);
    a = fma(z, a, 1.0 / 362880.0);
    b = fma(z, b, -1.0 / 3628800.0);
    a = fma(z, a, -1.0 / 5040.0);
    b = fma(z, b, 1.0 / 40320.0);
    a = fma(z, a, 1.0 / 120.0);
    b = fma(z, b, -1.0 / 720.0);
    a = fma(z, a, -1.0 / 6.0);
    b = fma(z, b, 1.0 / 24.0);
    b = fma(z, b, -0.5);
    const double sy = fma(y * z, a, y), cy = fma(z, b, 1.0);
    // quadrant n mod 4: (s, c), (c, -s), (-s, -c), (-c, s)
    const double u = n & 1 ? cy : sy, v = n & 1 ? sy : cy;
    s = __hiloint2double(__double2hiint(u) ^ ((n & 2) << 30), __double2loint(u));
    c = __hiloint2double(__double2hiint(v) ^ (((n + 1) & 2) << 30), __double2loint(v));
    const unsigned at = (unsigned)__double2hiint(x) & 0x7fffffffu;
    if (LIB) {
        if (at >= kSinCosMax) sincos(x, &s, &c);
    } else {
        odd = max(odd, at);
    }
}

}  // namespace fmm
