// fp8 e4m3 block quantisation with power-of-two scales (UE8M0), the activation / weight format of the
// expert GEMMs: a block of 128 values shares one scale s = 2^e, the smallest power of two with
// amax / s <= 448. Such a scale is exactly the byte the block-scaled tensor-core MMA wants (its biased
// fp32 exponent), and multiplying or dividing by it is exact.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <stdint.h>

namespace mfk {

__device__ __forceinline__ float pow2_scale_e4m3(float amax)
{
    const uint32_t b = __float_as_uint(amax * (1.f / 448.f));
    uint32_t e = (b + 0x7FFFFFu) >> 23;  // amax > 0: the sign bit is clear; the scale is rounded up to the next power of two
    e = min(max(e, 1u), 254u);
    return amax > 0.f ? __uint_as_float(e << 23) : 1.f;  // a select: no branch in front of what follows
}

// The UE8M0 byte of a power-of-two fp32 scale.
__device__ __forceinline__ uint32_t ue8m0_byte(float scale) { return (__float_as_uint(scale) >> 23) & 0xFFu; }

// Four floats -> four e4m3 bytes (saturating), x[i] * mul.
__device__ __forceinline__ uint32_t pack4_e4m3(float a, float b, float c, float d, float mul)
{
    return (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(a * mul, b * mul), __NV_SATFINITE, __NV_E4M3) |
           ((uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(c * mul, d * mul), __NV_SATFINITE, __NV_E4M3) << 16);
}

// ---- bf16 rows ----------------------------------------------------------------------------------------
// The quantisers of bf16 rows are bound by their instructions, so they stay with pairs of bf16 as long as that is exact: maxima of magnitudes are, and
// so is the product with a power of two (what falls below bf16's normal range is far below half of e4m3's smallest value). The bytes are
// those of pack4_e4m3(x, 1 / scale).

// Largest magnitudes of eight bf16, in two halves; a NaN counts as nothing.
__device__ __forceinline__ __nv_bfloat162 amax_bf16(const uint4 &v)
{
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&v);
    return __hmax2(__hmax2(__habs2(h[0]), __habs2(h[1])), __hmax2(__habs2(h[2]), __habs2(h[3])));
}
__device__ __forceinline__ __nv_bfloat162 shfl_xor_bf162(__nv_bfloat162 v, int o)
{
    const uint32_t got = __shfl_xor_sync(0xffffffffu, *reinterpret_cast<uint32_t *>(&v), o);
    return *reinterpret_cast<const __nv_bfloat162 *>(&got);
}
__device__ __forceinline__ float amax_of(__nv_bfloat162 v)
{
    const float2 f = __bfloat1622float2(v);
    return fmaxf(fmaxf(f.x, f.y), 0.f);
}

// 1 / scale of a scale that pow2_scale_e4m3 gives, twice as bf16 (a power of two; 2^-127 is subnormal).
__device__ __forceinline__ __nv_bfloat162 inverse_bf162(float scale)
{
    const uint32_t b = max(0x7F000000u - __float_as_uint(scale), 0x00400000u) >> 16;
    const uint32_t two = b | (b << 16);
    return *reinterpret_cast<const __nv_bfloat162 *>(&two);
}

// Eight bf16 times `mul` as e4m3 (saturating).
__device__ __forceinline__ uint2 pack8_e4m3(const uint4 &v, __nv_bfloat162 mul)
{
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&v);
    uint32_t q[4];
#pragma unroll
    for (int i = 0; i < 4; i++) q[i] = __nv_cvt_float2_to_fp8x2(__bfloat1622float2(__hmul2(h[i], mul)), __NV_SATFINITE, __NV_E4M3);
    return make_uint2(q[0] | (q[1] << 16), q[2] | (q[3] << 16));
}

}  // namespace mfk
