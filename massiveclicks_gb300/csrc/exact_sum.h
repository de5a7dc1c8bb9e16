// Sums of floats as 64-bit integers.  An FP64 add and its conversion go at two a
// cycle for an SM, so that a sum of many FP32 terms is bound by them; a pair of
// floats is as fast as this and keeps 48 bits.  A term here is its 24-bit
// significand shifted to the unit of the sum's largest term: FP64 sums of the same
// terms round at 2^-53 of the sum, this at 2^-55 of the largest term, and not at
// all for terms within 2^32 of it.
#ifndef MCLICKS_EXACT_SUM_H
#define MCLICKS_EXACT_SUM_H

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define MC_HD __host__ __device__ __forceinline__
#else
#define MC_HD inline
#endif

namespace mcd {

// A finite float >= 0 (bits u) in units of 2^(top - 182), top at least its
// exponent field.  256 terms fit in 64 bits.  Subnormal terms are left out.
MC_HD uint64_t fixed_term(uint32_t u, uint32_t top) {
    const uint32_t e = u >> 23, d = top - e;
    const uint32_t m = e ? (u & 0x7FFFFFu) | 0x800000u : 0u;
    return ((uint64_t)m << 32) >> (d < 63u ? d : 63u);
}

// The value of a sum of terms, rounded once.
MC_HD double fixed_value(uint64_t sum, uint32_t top) {
    const uint64_t bits = (uint64_t)(top + 841u) << 52;  // 2^(top - 182)
    double unit;
    memcpy(&unit, &bits, sizeof unit);
    return (double)sum * unit;
}

}  // namespace mcd

#endif
