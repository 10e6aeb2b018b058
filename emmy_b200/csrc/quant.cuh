// Codes of eight 16-bit activations divided by one scale, for the activation quantizers of the FP8 and NVFP4 linears.
//
// The rule divides every element by the scale in f32, rounds to nearest, and encodes the quotient (round to nearest even, saturating).
// Encoding is monotonic, so a division per element is not needed: with lo <= 1 / s <= hi a hair apart (one division per
// scale), fl(v lo) and fl(v hi) enclose fl(v / s) on either side of zero, and where both encode to the same code that is the code
// of the quotient.  Where an element's two codes differ the quotient lies within 2^-20, relatively, of a rounding boundary, and is
// divided.  With a scale that comes from a maximum of 16-bit values that is not rare: quotients of short significands often fall on a
// boundary (e2m1, 1024 x 5120 normal bf16 values with a maximum of 5.0625: 0.4 % of the elements, so 3 % of the groups of eight and 85 %
// of the warps).
//
// So e2m1 divides only the elements concerned.  Measured against dividing the group of eight, us an NVFP4 linear of K=5120, rows x columns: bf16
// 300 x 5120 17.9 -> 17.1, 2048 x 2048 22.0 -> 20.5, f16 2048 x 2048 20.0 -> 19.8 (sixteen elements in one loop: f16 21.0).
// e4m3 divides the group: looking for the element gave nothing (FP8 linear of 128 rows 25.6 and 26.0 us).
#pragma once
#include "common.cuh"

namespace eq {
namespace quant {

__device__ __forceinline__ uint32_t e4m3x2(float lo, float hi) {
    uint16_t r;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));  // first source -> upper byte
    return r;
}
// two f32 -> one byte: low nibble = code(lo), high nibble = code(hi)
__device__ __forceinline__ uint32_t e2m1x2(float lo, float hi) {
    uint16_t r;
    asm("{ .reg .b8 t; cvt.rn.satfinite.e2m1x2.f32 t, %1, %2; cvt.u16.u8 %0, t; }" : "=h"(r) : "f"(hi), "f"(lo));
    return r;
}

// 1 / s from below and from above, with room for the rounding of the reciprocal and of this product; false where s is so large
// (or not a number) that the reciprocal would lose bits.
__device__ __forceinline__ bool bracket(float s, float& lo, float& hi) {
    const float r = __fdiv_rn(1.0f, s);
    lo = __fmul_rn(r, 1.0f - 0x1p-21f);
    hi = __fmul_rn(r, 1.0f + 0x1p-21f);
    return s < 0x1p100f;
}

// max |v| of eight values; NaNs do not count.
template <typename InT>
__device__ __forceinline__ float abs_max8(const uint4& raw);
template <>
__device__ __forceinline__ float abs_max8<__half>(const uint4& raw) {
    auto mag = [](uint32_t w) { w &= 0x7FFF7FFFu; return *reinterpret_cast<const __half2*>(&w); };
    const __half2 m = __hmax2(__hmax2(mag(raw.x), mag(raw.y)), __hmax2(mag(raw.z), mag(raw.w)));
    return fmaxf(0.f, fmaxf(__low2float(m), __high2float(m)));
}
template <>
__device__ __forceinline__ float abs_max8<__nv_bfloat16>(const uint4& raw) {
    auto mag = [](uint32_t w) { w &= 0x7FFF7FFFu; return *reinterpret_cast<const __nv_bfloat162*>(&w); };
    const __nv_bfloat162 m = __hmax2(__hmax2(mag(raw.x), mag(raw.y)), __hmax2(mag(raw.z), mag(raw.w)));
    return fmaxf(0.f, fmaxf(__low2float(m), __high2float(m)));
}

// e4m3(v / s) of eight values.
template <typename InT>
__device__ __forceinline__ uint2 e4m3_codes8(const uint4& raw, float s) {
    const InT* e = reinterpret_cast<const InT*>(&raw);
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = to_float(e[i]);
    float lo, hi;
    if (bracket(s, lo, hi)) {
        uint32_t a[2], b[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            a[h] = e4m3x2(__fmul_rn(v[4 * h], lo), __fmul_rn(v[4 * h + 1], lo)) | (e4m3x2(__fmul_rn(v[4 * h + 2], lo), __fmul_rn(v[4 * h + 3], lo)) << 16);
            b[h] = e4m3x2(__fmul_rn(v[4 * h], hi), __fmul_rn(v[4 * h + 1], hi)) | (e4m3x2(__fmul_rn(v[4 * h + 2], hi), __fmul_rn(v[4 * h + 3], hi)) << 16);
        }
        if (a[0] == b[0] && a[1] == b[1]) return make_uint2(a[0], a[1]);
    }
    uint32_t w[2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
        w[h] = e4m3x2(__fdiv_rn(v[4 * h], s), __fdiv_rn(v[4 * h + 1], s)) | (e4m3x2(__fdiv_rn(v[4 * h + 2], s), __fdiv_rn(v[4 * h + 3], s)) << 16);
    return make_uint2(w[0], w[1]);
}

// The i-th (0 to 7) of eight values; for an i that only the running thread knows.
template <typename InT>
__device__ __forceinline__ float element8(const uint4& raw, int i) {
    const uint32_t w = i & 4 ? (i & 2 ? raw.w : raw.z) : (i & 2 ? raw.y : raw.x);
    const uint16_t h = static_cast<uint16_t>(i & 1 ? w >> 16 : w);
    return to_float(*reinterpret_cast<const InT*>(&h));
}

// e2m1(v / s) of eight values, two codes a byte.
template <typename InT>
__device__ __forceinline__ uint32_t e2m1_codes8(const uint4& raw, float s) {
    const InT* e = reinterpret_cast<const InT*>(&raw);
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = to_float(e[i]);
    float lo, hi;
    if (bracket(s, lo, hi)) {
        uint32_t a = 0, b = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            a |= e2m1x2(__fmul_rn(v[2 * i], lo), __fmul_rn(v[2 * i + 1], lo)) << (8 * i);
            b |= e2m1x2(__fmul_rn(v[2 * i], hi), __fmul_rn(v[2 * i + 1], hi)) << (8 * i);
        }
        for (uint32_t d = a ^ b; d;) {
            const int i = (__ffs(d) - 1) >> 2;
            const uint32_t mask = 0xFu << (4 * i);
            a = (a & ~mask) | ((e2m1x2(__fdiv_rn(element8<InT>(raw, i), s), 0.f) << (4 * i)) & mask);
            d &= ~mask;
        }
        return a;
    }
    uint32_t w = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) w |= e2m1x2(__fdiv_rn(v[2 * i], s), __fdiv_rn(v[2 * i + 1], s)) << (8 * i);
    return w;
}

}  // namespace quant
}  // namespace eq
