// FP32 and FP64 numbers into one another without the FP64 unit.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace semo {

// An FP32 number as a double, by integer instructions: the conversion
// instruction takes longer in the FP64 unit than a multiply-add (k_outer_mv at
// 128^3: 83 us, 48 with the integers, 37 without any FP64 arithmetic).  Every value, subnormal, infinite and
// not-a-number ones too.
__host__ __device__ __forceinline__ uint64_t wide_bits(uint32_t b) {
    const uint32_t sign = b & 0x80000000u, m = b & 0x7fffffu, e = (b >> 23) & 0xffu;
    // exponents: 127 -> 1023, 255 -> 2047
    uint32_t hi = sign | (((b & 0x7fffffffu) >> 3) + (e == 255 ? 0x70000000u : 0x38000000u));
    uint32_t lo = b << 29;
    if (e == 0) {   // zero or subnormal: m 2^-149
        hi = sign;
        lo = 0;
#pragma unroll 1
        for (uint32_t k = m, x = 896; k != 0; k <<= 1, --x)
            if (k & 0x400000u) {   // the leading bit becomes the implicit one
                hi = sign | (x << 20) | ((k & 0x3fffffu) >> 2);
                lo = k << 30;
                break;
            }
    }
    return ((uint64_t)hi << 32) | lo;
}
// (float)d by integer instructions, rounded to nearest even, for the same reason
__host__ __device__ __forceinline__ uint32_t narrow_bits(uint64_t u) {
    const uint32_t sign = (uint32_t)(u >> 32) & 0x80000000u, e = (uint32_t)(u >> 52) & 0x7ffu;
    if (e - 897u <= 253u) {   // in the range of normal FP32 numbers
        const uint32_t t = (uint32_t)((u & 0x7fffffffffffffffull) >> 29) - (896u << 23);
        const uint32_t rest = (uint32_t)u & 0x1fffffffu;
        return sign | (t + (rest > 0x10000000u - (t & 1u) ? 1u : 0u));
    }
    if (e == 0x7ff && (u & 0xfffffffffffffull)) return sign | 0x7fc00000u;
    if (e > 1150u) return sign | 0x7f800000u;
    if (e < 872u) return sign;   // below half the smallest subnormal
    const uint64_t m = (u & 0xfffffffffffffull) | 0x10000000000000ull;
    const int sh = 29 + (int)(897u - e);   // 30 .. 54
    const uint64_t t = m >> sh, rest = m & ((1ull << sh) - 1), half = 1ull << (sh - 1);
    return sign | (uint32_t)(t + (rest > half || (rest == half && (t & 1)) ? 1 : 0));
}
template <class V>
__device__ __forceinline__ V narrow(double d) {
    if constexpr (sizeof(V) == 4) return __uint_as_float(narrow_bits((uint64_t)__double_as_longlong(d)));
    else return d;
}
template <class V, class X>
__device__ __forceinline__ V widen(X x) {
    if constexpr (sizeof(V) > sizeof(X)) return __longlong_as_double((long long)wide_bits(__float_as_uint(x)));
    else return x;
}

}  // namespace semo
