// FP64 <-> FP32-pair conversions on bit patterns, for the host and the device.
//
// A conversion between double and float issues on the FP64 pipe (1/64 of the FP32 rate here): with two
// conversions and a subtraction per entry the split of 34.5 M entries took 0.24 ms against 0.08 ms for
// its memory traffic.  These work on the bit patterns instead (of tiny entries too: products of 1D
// coefficients that are rounding noise reach far below the FP32 range).  The results are the same bits
// (tests/pair_bits_check.cu compares them).
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>

namespace amdg {

__host__ __device__ __forceinline__ uint64_t bits_of(double v) {
#ifdef __CUDA_ARCH__
    return uint64_t(__double_as_longlong(v));
#else
    uint64_t b;
    std::memcpy(&b, &v, sizeof(b));
    return b;
#endif
}
__host__ __device__ __forceinline__ uint32_t bits_of(float v) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(v);
#else
    uint32_t b;
    std::memcpy(&b, &v, sizeof(b));
    return b;
#endif
}
__host__ __device__ __forceinline__ double double_of(uint64_t b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double v;
    std::memcpy(&v, &b, sizeof(v));
    return v;
#endif
}
__host__ __device__ __forceinline__ float float_of(uint32_t b) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float v;
    std::memcpy(&v, &b, sizeof(v));
    return v;
#endif
}
__host__ __device__ __forceinline__ int leading_zeros(uint32_t b) {
#ifdef __CUDA_ARCH__
    return __clz(int(b));
#else
    return b ? __builtin_clz(b) : 32;
#endif
}

// the conversions themselves, out of line: inlined, the compiler issues them for every entry and selects
static __host__ __device__ __noinline__ float2 split_convert(double d) {
    const float h = float(d);
    return make_float2(h, float(d - double(h)));
}
static __host__ __device__ __noinline__ double widen_convert(float f) { return double(f); }

// float(v), |v| <= 2^28, without a conversion: two exact parts through the mantissa of 1.5 * 2^23, one
// rounding in the multiply-add
__host__ __device__ __forceinline__ float small_to_float(int v) {
    const float a = float_of(0x4b400000u + uint32_t(v >> 14)) - 12582912.0f;
    const float b = float_of(0x4b400000u + uint32_t(v & 0x3fff)) - 12582912.0f;
    return fmaf(a, 16384.0f, b);
}

// hi = float(d), lo = float(d - hi), both rounded to nearest even
__host__ __device__ __forceinline__ void split_bits(double d, float& hi, float& lo) {
    const uint64_t b = bits_of(d);
    const int e = int(b >> 52) & 0x7ff;
    const uint32_t sign = uint32_t(b >> 32) & 0x80000000u;
    if (e < 1023 - 126) {  // below the normal floats: multiples of 2^-149, what is left rounds to zero
        const uint64_t mant = (b & 0xfffffffffffffull) | (e ? 0x10000000000000ull : 0);
        const int s = 1023 - 97 - (e ? e : 1);  // 2^-149 in units of mant's last bit, 30 or more
        uint64_t keep = 0, rem = mant;
        if (s < 54) {
            keep = mant >> s;
            rem = mant & ((1ull << s) - 1);
            const uint64_t half = 1ull << (s - 1);
            if (rem > half || (rem == half && (keep & 1))) {
                ++keep;
                hi = float_of(sign | uint32_t(keep));
                lo = float_of(sign ^ 0x80000000u);  // d - hi points back to zero
                return;
            }
        }
        hi = float_of(sign | uint32_t(keep));
        lo = float_of(rem ? sign : 0u);
        return;
    }
    if (e > 1023 + 126) {  // may round up to infinity, or is not finite
        const float2 p = split_convert(d);
        hi = p.x;
        lo = p.y;
        return;
    }
    const uint64_t mant = (b & 0xfffffffffffffull) | 0x10000000000000ull;
    uint32_t keep = uint32_t(mant >> 29);                   // 24 bits, the leading one included
    const uint32_t rem = uint32_t(mant) & 0x1fffffffu;      // 29 bits
    const bool up = rem > 0x10000000u || (rem == 0x10000000u && (keep & 1u));
    keep += up ? 1u : 0u;
    hi = float_of(sign | ((uint32_t(e - 1023 + 126) << 23) + keep));
    int diff = int(rem) - (up ? 0x20000000 : 0);            // d - hi in units of 2^s
    int s = e - 1023 - 52;
    if (s < -149) {
        // the unit is below the smallest float: round to the coarser of it and 24 bits
        const uint32_t a = uint32_t(diff < 0 ? -diff : diff);
        const int wide = a ? 8 - leading_zeros(a) : 0, drop = -149 - s > wide ? -149 - s : wide;
        uint32_t q = a >> drop;
        const uint32_t r = a & ((1u << drop) - 1u), half = 1u << (drop - 1);
        q += r > half || (r == half && (q & 1u)) ? 1u : 0u;
        const bool zero = a == 0;
        const uint32_t lsign = zero ? 0u : (sign ^ (diff < 0 ? 0x80000000u : 0u));
        s += drop;
        lo = float_of(lsign | bits_of(small_to_float(int(q)) * float_of(s >= -126 ? uint32_t(s + 127) << 23 : 1u << (s + 149))));
        return;
    }
    diff = sign ? -diff : diff;
    lo = small_to_float(diff) * float_of(s >= -126 ? uint32_t(s + 127) << 23 : 1u << (s + 149));  // exact
}

// double(f)
__host__ __device__ __forceinline__ double widen_bits(float f) {
    const uint32_t b = bits_of(f);
    const uint32_t e = (b >> 23) & 0xffu, m = b & 0x7fffffu;
    if (e == 0xffu) return widen_convert(f);
    uint64_t w = 0;
    if (e) {
        w = (uint64_t(e + (1023 - 127)) << 52) | (uint64_t(m) << 29);
    } else if (m) {  // m * 2^-149
        const int n = 31 - leading_zeros(m);
        w = (uint64_t(1023 - 149 + n) << 52) | ((uint64_t(m) << (52 - n)) & 0xfffffffffffffull);
    }
    return double_of((uint64_t(b & 0x80000000u) << 32) | w);
}

}  // namespace amdg
