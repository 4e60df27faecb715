// GGUF quants and f32 activations as f16 operands, shared by the dequantising products.
//
// Eight consecutive elements travel together.  Their order is the natural one for Q8_0 and 0 4 1 5 2 6 3 7 for Q4_0, in which the
// nibbles of a word come out of it; both operands use the same order, so that the products do not change.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

__device__ __forceinline__ uint32_t gguf_sub_f16(uint32_t v, uint32_t offset)
{
    const __half2 r = __hsub2(*reinterpret_cast<const __half2 *>(&v), *reinterpret_cast<const __half2 *>(&offset));
    return *reinterpret_cast<const uint32_t *>(&r);
}
// the eight nibbles of a word, minus 8 (0x6400 is 1024 in f16: a nibble becomes its last bits)
__device__ __forceinline__ void gguf_nibbles_f16(uint32_t w, uint32_t (&h)[4])
{
#pragma unroll
    for (int i = 0; i < 4; i++) h[i] = gguf_sub_f16(((w >> (4 * i)) & 0x000f000fu) | 0x64006400u, 0x64086408u);
}
// eight signed bytes
__device__ __forceinline__ void gguf_bytes_f16(uint32_t lo, uint32_t hi, uint32_t (&h)[4])
{
    lo ^= 0x80808080u;
    hi ^= 0x80808080u;
    h[0] = gguf_sub_f16(__byte_perm(lo, 0x64646464u, 0x4140), 0x64806480u);
    h[1] = gguf_sub_f16(__byte_perm(lo, 0x64646464u, 0x4342), 0x64806480u);
    h[2] = gguf_sub_f16(__byte_perm(hi, 0x64646464u, 0x4140), 0x64806480u);
    h[3] = gguf_sub_f16(__byte_perm(hi, 0x64646464u, 0x4342), 0x64806480u);
}
// exponent e of the largest element: x * 2^(14 - e) is below 2^15 and both factors are normal numbers
__device__ __forceinline__ int gguf_exponent(float largest) { return largest > 0.0f && largest < INFINITY ? max(-110, ilogbf(largest)) : 0; }
// v * scale = h1 + h2, two f16 numbers: 22 significant bits, or 2^-39 of the largest element where that is more.  An element that is
// not finite gives h2 = NaN.
template <bool Q4>
__device__ __forceinline__ void gguf_split8(const float (&v)[8], float scale, uint4 &h1, uint4 &h2)
{
    uint32_t p1[4], p2[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float a = v[Q4 ? i : 2 * i] * scale, b = v[Q4 ? i + 4 : 2 * i + 1] * scale;
        const __half2 h = __floats2half2_rn(a, b);
        const float2 f = __half22float2(h);
        const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
        p1[i] = *reinterpret_cast<const uint32_t *>(&h);
        p2[i] = *reinterpret_cast<const uint32_t *>(&l);
    }
    h1 = make_uint4(p1[0], p1[1], p1[2], p1[3]);
    h2 = make_uint4(p2[0], p2[1], p2[2], p2[3]);
}
