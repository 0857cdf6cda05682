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
// |v| between 2^-900 and 2^900 (exponent fields 123 and 1923)
SPH_HD bool mid_range(uint64_t u) { return ((uint32_t)(u >> 52) & 0x7ffu) - 123u < 1800u; }

// Quotients x / b of many values by one, correctly rounded: x rb (rb = 1 / b
// rounded) and two residual corrections, of which the first brings it within
// one unit in the last place and the second rounds it as the division does
// (Markstein, IBM J. Res. Dev. 34, 1990, on the final rounding of a quotient):
// 5 FP64 operations instead of about 9, of which an SM has two lanes.  That
// needs exact residuals and normal numbers: true where *q is the quotient,
// false where the caller has to divide (operands or quotients outside 2^-900
// to 2^900, infinities, NaN).
struct Divisor {
    double b, rb;
};
SPH_HD Divisor divisor(double b)
{
    // (a NaN for rb makes every quotient the caller's)
    return Divisor{b, mid_range(bits_of(b)) ? 1.0 / b : std::nan("")};
}
SPH_HD bool quotient(double x, const Divisor& d, double* q)
{
    const double q0 = x * d.rb;
    const double q1 = fma_rn(fma_rn(-q0, d.b, x), d.rb, q0);
    const double q2 = fma_rn(fma_rn(-q1, d.b, x), d.rb, q1);
    const bool zero = (bits_of(x) << 1) == 0;  // x rb has its sign
    *q = zero ? q0 : q2;
    return zero ? d.rb == d.rb : (mid_range(bits_of(x)) && mid_range(bits_of(q2)));
}

}  // namespace sph
