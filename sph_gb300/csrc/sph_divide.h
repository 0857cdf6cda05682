// Division of many values by one.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define SPH_HD __host__ __device__ __forceinline__
#else
#define SPH_HD inline
#endif

namespace sph {

SPH_HD double fma_rn(double a, double b, double c)
{
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
SPH_HD uint64_t bits_of(double v)
{
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t u;
    std::memcpy(&u, &v, 8);
    return u;
#endif
}
// Quotients x / b of many values by one, correctly rounded: the product of x
// with 1 / b in two parts, which is within one unit in the last place of the
// quotient, and one residual correction, which rounds it as the division does
// (Markstein, IBM J. Res. Dev. 34, 1990, on the final rounding of a quotient):
// 4 FP64 operations instead of about 9, of which an SM has two lanes.  That
// needs exact residuals and normal numbers: true where *q is the quotient,
// false where the caller has to divide (|b| outside 2^-100 to 2^100; |x|
// outside 2^-800 to 2^800 but zero).
struct Divisor {
    double b, hi, lo;  // 1 / b rounded, and what that left out
    bool ok;
};
SPH_HD Divisor divisor(double b)
{
    const bool ok = ((uint32_t)(bits_of(b) >> 52) & 0x7ffu) - 923u < 200u;
    const double hi = 1.0 / b;
    return Divisor{b, hi, fma_rn(-hi, b, 1.0) * hi, ok};
}
SPH_HD bool quotient(double x, const Divisor& d, double* q)
{
    const double q0 = fma_rn(x, d.hi, x * d.lo);
    const double q1 = fma_rn(fma_rn(-q0, d.b, x), d.hi, q0);
    *q = q1;
    // a zero (of either sign) gives a zero
    const uint64_t u = bits_of(x);
    return d.ok && (((uint32_t)(u >> 52) & 0x7ffu) - 223u < 1600u || (u << 1) == 0);
}

}  // namespace sph
