// mdt_convert.h -- FP64 <-> FP32 conversions by integer instructions.  The conversion instructions run
// on the FP64 pipe of sm_103a (55 cycles a warp, an integer instruction 1-2).  Results are theirs, bit
// for bit: rounded to nearest, halves to even, denormals, infinities; any NaN gives a quiet NaN.
// Plain C++ as well, so that they can be compared with the casts on the host.
#pragma once
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define MDT_CONVERT static __host__ __device__ __forceinline__
#else
#define MDT_CONVERT static inline
#endif

namespace mdt {

MDT_CONVERT uint64_t bits_of(double x) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return u;
#endif
}

MDT_CONVERT float float_of_bits(uint32_t u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    std::memcpy(&f, &u, 4);
    return f;
#endif
}

MDT_CONVERT uint32_t bits_of(float f) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(f);
#else
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return u;
#endif
}

MDT_CONVERT double double_of_bits(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t u = (uint64_t)hi << 32 | lo;
    double x;
    std::memcpy(&x, &u, 8);
    return x;
#endif
}

// (float)x where the result is 0 or normal
MDT_CONVERT float f32_normal(double x) {
    const uint64_t u = bits_of(x);
    const uint32_t hi = (uint32_t)(u >> 32), lo = (uint32_t)u;
    const uint32_t m = ((hi << 3 | lo >> 29) ^ 0x40000000u) & 0x7fffffffu;
    const uint32_t v = m + (((lo & 0x1fffffffu) + 0x0fffffffu + (m & 1u)) >> 29);
    return float_of_bits(((hi & 0x7ff00000u) < 0x38100000u ? 0u : v) | (hi & 0x80000000u));
}

// Neither 0 nor a normal FP32 number: the cast itself, as a call, because inlined it costs the
// registers of every kernel that converts.
#ifdef __CUDACC__
static __host__ __device__ __noinline__ float f32_rare(double x) { return (float)x; }
#else
static inline float f32_rare(double x) { return (float)x; }
#endif

// (float)x
MDT_CONVERT float f32_of(double x) {
    const uint64_t a = bits_of(x) & 0x7fffffffffffffffull;
    if ((uint32_t)(a >> 32) - 0x38100000u >= 0x0fe00000u && a != 0) return f32_rare(x);
    return f32_normal(x);
}

// (double)f
MDT_CONVERT double f64_of(float f) {
    // a denormal times 2^64 is normal, and exact
    const bool tiny = (bits_of(f) & 0x7f800000u) == 0;
    const uint32_t u = bits_of(tiny ? f * 0x1p64f : f), m = u & 0x7fffffffu;
    uint32_t h = (m >> 3) + (tiny ? 0x34000000u : 0x38000000u);
    if (m == 0) h = 0u;
    if (m >= 0x7f800000u) h = m > 0x7f800000u ? 0x7fffffffu : 0x7ff00000u;
    return double_of_bits(h | (u & 0x80000000u), u << 29);
}

// x = h + l to 48 bits: h = (float)x, l = (float)(x - h).  From 2^-72 up to 2^127 neither part is
// denormal (the last place of x is 2^-124 or more).
MDT_CONVERT bool splits_normal(double x) {
    const uint64_t a = bits_of(x) & 0x7fffffffffffffffull;
    return (uint32_t)(a >> 32) - 0x3b700000u < 0x0c700000u || a == 0;
}
MDT_CONVERT void split_normal(double x, float &h, float &l) {
    h = f32_normal(x);
    l = f32_normal(x - f64_of(h));
}

// the hi/lo split of a position
MDT_CONVERT void split3(double x, double y, double z, float (&h)[3], float (&l)[3]) {
    if (splits_normal(x) && splits_normal(y) && splits_normal(z)) {
        split_normal(x, h[0], l[0]);
        split_normal(y, h[1], l[1]);
        split_normal(z, h[2], l[2]);
    } else {
        h[0] = (float)x;
        h[1] = (float)y;
        h[2] = (float)z;
        l[0] = (float)(x - (double)h[0]);
        l[1] = (float)(y - (double)h[1]);
        l[2] = (float)(z - (double)h[2]);
    }
}

}  // namespace mdt
