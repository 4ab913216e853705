// Correctly rounded FP64 quotients by one divisor, given the rounded
// reciprocal of that divisor: a cell divides many sums by its volume, and
// after the one IEEE division 1 / b each further quotient takes five
// multiply / FMA operations instead of a full division.  Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor" (1990); the
// statement used here is that of Muller et al., Handbook of Floating-Point
// Arithmetic (division with an FMA): with y = RN(1/b), a faithful quotient q
// and the exact remainder r = a - b q, RN(q + r y) is RN(a / b) as long as
// nothing over- or underflows.  The first correction makes q faithful, the
// second one makes it correctly rounded.  Operands outside the exponent range
// where every intermediate is normal (zeros, infinities and NaN among them)
// take the plain division, so the result is a / b bit for bit everywhere.
// Host and device: tests/rn_div_check.cpp compiles it for the host.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define ZSME_RNDIV_FN __host__ __device__ __forceinline__
#else
#define ZSME_RNDIV_FN inline
#endif

namespace zsme {

// upper word without the sign: the biased exponent in its top 11 bits
ZSME_RNDIV_FN uint32_t exponent_word(double a) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2hiint(a) & 0x7fffffffu;
#else
    uint64_t u;
    std::memcpy(&u, &a, sizeof u);
    return (uint32_t)(u >> 32) & 0x7fffffffu;
#endif
}
ZSME_RNDIV_FN uint32_t lower_word(double a) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2loint(a);
#else
    uint64_t u;
    std::memcpy(&u, &a, sizeof u);
    return (uint32_t)u;
#endif
}
ZSME_RNDIV_FN double rn_fma(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}

// RN(1 / b) for |b| in [2^-100, 2^100) without a branch: Newton-Raphson from a
// seed good to 2^-18 or better (two steps reach half an ulp and a bit, the
// third rounds correctly by Markstein's theorem on reciprocals, which leaves
// out the significand of all ones).  odd is set where b is outside that range
// or may have that significand.
ZSME_RNDIV_FN double rn_reciprocal(double b, bool& odd) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
#else
    double y = (double)(1.0f / (float)b) * (1.0 + 0x1p-19);
#endif
    odd |= (exponent_word(b) - (923u << 20) >= (200u << 20)) | (lower_word(b) == 0xffffffffu);
    y = rn_fma(rn_fma(-b, y, 1.0), y, y);
    y = rn_fma(rn_fma(-b, y, 1.0), y, y);
    return rn_fma(rn_fma(-b, y, 1.0), y, y);
}

struct RnDivisor {
    double b, y;
    // the plain division serves every quotient where |b| is not in [2^-100, 2^100)
    bool fast;
    ZSME_RNDIV_FN explicit RnDivisor(double div)
        : b(div), y(1.0 / div), fast(exponent_word(div) - (923u << 20) < (200u << 20)) {}
    ZSME_RNDIV_FN RnDivisor(double div, double reciprocal)   // reciprocal: 1 / div, formed before
        : b(div), y(reciprocal), fast(exponent_word(div) - (923u << 20) < (200u << 20)) {}
    ZSME_RNDIV_FN double quotient(double a) const {
        const double q0 = a * y;
        const double q1 = rn_fma(rn_fma(-b, q0, a), y, q0);
        double q = rn_fma(rn_fma(-b, q1, a), y, q1);
        // |a| outside [2^-900, 2^900): q is not to be trusted; of a zero, q0 has the sign
        if (!fast || exponent_word(a) - (123u << 20) >= (1800u << 20)) q = (fast && a == 0.0) ? q0 : a / b;
        return q;
    }
    // The same without a branch, for b > 0 and an a that is never a negative zero: where the
    // five operations do not give the quotient, odd is set and the caller
    // divides again.
    ZSME_RNDIV_FN double quotient_or(double a, bool& odd) const {
        const double q0 = a * y;
        const double q1 = rn_fma(rn_fma(-b, q0, a), y, q0);
        const uint32_t e = exponent_word(a);
        odd |= !fast | ((e - (123u << 20) >= (1800u << 20)) & ((e | lower_word(a)) != 0u));
        return rn_fma(rn_fma(-b, q1, a), y, q1);
    }
    // quotient_or for any b and a
    ZSME_RNDIV_FN double signed_quotient_or(double a, bool& odd) const {
        const double q = quotient_or(a, odd);
        return a == 0.0 ? a * y : q;
    }
};

// a[i] /= b for every i
template <int N>
ZSME_RNDIV_FN void divide_all(double (&a)[N], double b) {
    const RnDivisor by(b);
    bool odd = false;
    double q[N];
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int i = 0; i < N; ++i) q[i] = by.signed_quotient_or(a[i], odd);
    if (odd) {
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int i = 0; i < N; ++i) q[i] = a[i] / b;
    }
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int i = 0; i < N; ++i) a[i] = q[i];
}

}  // namespace zsme
