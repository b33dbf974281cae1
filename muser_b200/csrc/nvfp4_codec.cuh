// The NVFP4 activation codec shared by the quantizer kernels and by the GEMM epilogue that emits quantized outputs:
// quant::activation_group_codes (crates/muser-engine/src/quant/nvfp4.rs:173-217), bit for bit.
#pragma once
#include <cuda_fp8.h>

#include "common.cuh"

namespace muser {

// Eight magnitudes-with-sign -> one word of E2M1 codes, the first in the low nibble: nearest, ties to the even code,
// saturating, the sign of a zero kept.
__device__ __forceinline__ uint32_t e2m1_word(const float (&q)[8]) {
    uint32_t w;
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
        "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
        : "=r"(w) : "f"(q[0]), "f"(q[1]), "f"(q[2]), "f"(q[3]), "f"(q[4]), "f"(q[5]), "f"(q[6]), "f"(q[7]));
    return w;
}

// Quantizes one group of 16 values: its 8 code bytes (as two words, or written), and its E4M3 scale code as the result.
//
// The reference compares m = |r| * isi with scale * {0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5} by > and >= in turn.  Those
// products are exact (a 4-bit and a 3-bit significand), the bounds are the midpoints between neighbouring E2M1 values
// and the >= ones belong to the even code: the chain is "m / scale to the nearest E2M1 value, ties to even", which is
// one conversion instruction.  The quotient has to be the correctly rounded one: two floats m and scale * bound that
// differ, differ by more than half a unit of the bound's last place after the division, so the rounded quotient meets a
// midpoint only where m met it.  It is made without a divide, by the residual of a product with the rounded
// reciprocal (tests/test_nvfp4_codec_cpu.py runs every scale against the floats around every bound).  The chain (seven
// multiplies, compares and adds a value) bounded both quantizer kernels and the GEMM epilogue that quantizes: quantize
// of 32768 x 5120 237 -> 117 us (the memory alone: 66; 79 with four rows a thread), behind the norm 334 -> 227, gate/up + quantize 6.14 -> 4.82 ms.
__device__ __forceinline__ uint32_t quantize_group(const float (&r)[16], float isi, uint32_t &codes_lo, uint32_t &codes_hi) {
    __half2 h[8], top = __floats2half2_rn(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        h[i] = __floats2half2_rn(r[2 * i], r[2 * i + 1]);
        top = __hmax2_nan(top, __habs2(h[i]));
    }
    const float2 top2 = __half22float2(top);
    float amax = fmaxf(top2.x, top2.y);
    float m[16], v[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float2 f = __half22float2(h[i]);
        v[2 * i] = f.x, v[2 * i + 1] = f.y;
        m[2 * i] = __fmul_rn(fabsf(f.x), isi), m[2 * i + 1] = __fmul_rn(fabsf(f.y), isi);
    }
    // A NaN is left out of the maximum and compares false all along (code 0 with its sign); an infinity, or a product
    // that overflows, is above every bound: the former become 0, the latter a number that still is.
    if (!(__fmul_rn(top2.x, isi) <= 1e30f && __fmul_rn(top2.y, isi) <= 1e30f)) {
        amax = 0.0f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            amax = fmaxf(amax, fabsf(v[i]));
            m[i] = m[i] > 0.0f ? fminf(m[i], 1e30f) : 0.0f;
        }
    }
    const float target = fminf(__fmul_rn(__fmul_rn(amax, 1.0f / 6.0f), isi), 448.0f);
    const uint32_t scale_code = __nv_cvt_float_to_fp8(target, __NV_SATFINITE, __NV_E4M3) & 0x7Fu;
    const float scale = __half2float(__half(__nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)scale_code, __NV_E4M3)));
    const float inv = scale > 0.0f ? __frcp_rn(scale) : 0.0f; // no scale: only the signs remain
    float q[2][8];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float q0 = __fmul_rn(m[i], inv);
        const float q1 = __fmaf_rn(__fmaf_rn(-q0, scale, m[i]), inv, q0);
        q[i >> 3][i & 7] = __uint_as_float(__float_as_uint(q1) | (__float_as_uint(v[i]) & 0x80000000u));
    }
    codes_lo = e2m1_word(q[0]), codes_hi = e2m1_word(q[1]);
    return scale_code;
}
__device__ __forceinline__ uint32_t quantize_group(const float (&r)[16], float isi, uint8_t *codes) {
    uint32_t lo, hi;
    const uint32_t scale_code = quantize_group(r, isi, lo, hi);
    *reinterpret_cast<uint2 *>(codes) = make_uint2(lo, hi);
    return scale_code;
}

// Where the scale byte of (row, 16-value group grp) lives in the swizzled plane of a tensor with kt 64-value chunks
// per row (scripts/gx10/vllm/muser_vllm/exact_fp4_quant.py:149-162); the four groups of a chunk are consecutive bytes.
__device__ __forceinline__ size_t swizzled_scale_offset(uint32_t row, uint32_t grp, uint32_t kt) {
    return (size_t)(row / 128) * ((size_t)kt * 512) + (size_t)(grp / 4) * 512 + (row % 32) * 16 + ((row % 128) / 32) * 4 + grp % 4;
}

} // namespace muser
