// fcb_math.cuh -- exp / log with a fixed operation sequence.
//
// The exact Euler solver needs powers (p/pK)^((gamma-1)/(2 gamma)) etc.  These
// functions use only + - * / and bit manipulation, in one fixed order, so the
// FP64 path gives the same bits on every device and on the host (built without
// FMA contraction).  Method: Cody-Waite reduction by ln 2; log m = 2 atanh(s),
// s = (m-1)/(m+1), m in [1/sqrt2, sqrt2), series to s^23; exp r by its Taylor
// series to r^17 for |r| <= ln2/2.  Relative error below 4e-16 for normal
// arguments (log) and |y| < 700 (exp).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace fcb {

__device__ __forceinline__ double fcb_log(double x)
{
    const double LN2_HI = 6.93147180369123816490e-01, LN2_LO = 1.90821492927058770002e-10;
    const double SQRT2 = 1.41421356237309514547e+00;
    unsigned long long b = (unsigned long long)__double_as_longlong(x);
    int e = (int)((b >> 52) & 0x7ff) - 1023;
    b = (b & 0x000fffffffffffffULL) | 0x3ff0000000000000ULL;
    double m = __longlong_as_double((long long)b);
    if (m > SQRT2) { m = m * 0.5; e = e + 1; }
    const double s = (m - 1.0) / (m + 1.0);
    const double s2 = s * s;
    double p = 1.0 / 23.0;
    p = p * s2 + 1.0 / 21.0;
    p = p * s2 + 1.0 / 19.0;
    p = p * s2 + 1.0 / 17.0;
    p = p * s2 + 1.0 / 15.0;
    p = p * s2 + 1.0 / 13.0;
    p = p * s2 + 1.0 / 11.0;
    p = p * s2 + 1.0 / 9.0;
    p = p * s2 + 1.0 / 7.0;
    p = p * s2 + 1.0 / 5.0;
    p = p * s2 + 1.0 / 3.0;
    p = p * s2 + 1.0;
    const double lm = 2.0 * s * p;
    const double de = (double)e;
    return de * LN2_HI + (de * LN2_LO + lm);
}

// x / N, correctly rounded, for a small integer N, in a multiplication and an FMA instead of a
// division (Brisebarre, Muller and Raina, IEEE Trans. Computers 53, 2004): with zh = 1/N rounded
// and zl = 1/N - zh rounded, x/N is zh x + zl x to about 2^-53 ulp before the last rounding,
// and the quotient of a 53-bit number by N lies at least 1/(2N) ulp from the middle of two
// neighbouring numbers, so the rounding is that of the exact quotient.  (x well above the
// subnormal range; the sign of a zero is not kept.)  The exponential has twelve of these, and
// they were most of the exact Euler solver's FP64 time.
template <int N>
__device__ __forceinline__ double div_int(double x)
{
    if constexpr ((N & (N - 1)) == 0) {
        return x * (1.0 / N);
    } else {
        constexpr double zh = 1.0 / N;
        // 1 - N zh is exact: N zh is within 2^-53 of 1; split zh so that both products are exact
        constexpr double hi = (double)(float)zh, lo = zh - hi;
        constexpr double zl = ((1.0 - N * hi) - N * lo) / N;
        return fma(x, zh, x * zl);
    }
}

__device__ __forceinline__ double fcb_exp(double y)
{
    const double LN2_HI = 6.93147180369123816490e-01, LN2_LO = 1.90821492927058770002e-10;
    const double INV_LN2 = 1.44269504088896338700e+00;
    const double kd = floor(y * INV_LN2 + 0.5);
    const double r = (y - kd * LN2_HI) - kd * LN2_LO;
    double p = 1.0 + div_int<17>(r);
    p = 1.0 + div_int<16>(r) * p;
    p = 1.0 + div_int<15>(r) * p;
    p = 1.0 + div_int<14>(r) * p;
    p = 1.0 + div_int<13>(r) * p;
    p = 1.0 + div_int<12>(r) * p;
    p = 1.0 + div_int<11>(r) * p;
    p = 1.0 + div_int<10>(r) * p;
    p = 1.0 + div_int<9>(r) * p;
    p = 1.0 + div_int<8>(r) * p;
    p = 1.0 + div_int<7>(r) * p;
    p = 1.0 + div_int<6>(r) * p;
    p = 1.0 + div_int<5>(r) * p;
    p = 1.0 + div_int<4>(r) * p;
    p = 1.0 + div_int<3>(r) * p;
    p = 1.0 + div_int<2>(r) * p;
    p = 1.0 + r * p;
    const int k = (int)kd;
    const double scale = __longlong_as_double((long long)((unsigned long long)(k + 1023) << 52));
    return p * scale;
}

}  // namespace fcb
