// A float32 as three bfloat16: 8 + 8 + 8 bits of its significand, exact down to where the last part falls under bfloat16's range.
#pragma once
#include "common.cuh"

// x += y, two floats of a register pair at a time
__device__ __forceinline__ void add_pair(float& x0, float& x1, float y0, float y1) {
    asm("{\n .reg .b64 a, b;\n mov.b64 a, {%0, %1};\n mov.b64 b, {%2, %3};\n add.rn.f32x2 a, a, b;\n mov.b64 {%0, %1}, a;\n}" : "+f"(x0), "+f"(x1) : "f"(y0), "f"(y1));
}
// x -= a bfloat16 of the pair each, as it lies: no shift and no mask
__device__ __forceinline__ void less_part(float& x, float& y, uint32_t part) {
    asm("{\n .reg .b16 lo, hi, minus;\n mov.b32 {lo, hi}, %2;\n mov.b16 minus, 0xBF80;\n fma.rn.f32.bf16 %0, lo, minus, %0;\n fma.rn.f32.bf16 %1, hi, minus, %1;\n}"
        : "+f"(x), "+f"(y) : "r"(part));
}
// The parts of two floats as pairs of bfloat16; x and y are left with their third ones.  The first two are rounded to the nearest: the
// second is at most 2^-8 of the float, the third 2^-17 and of at most 7 bits, which lie in the upper halves; every subtraction is exact.
// What a product of two floats loses without the products of second and third parts is at most 2^-24 of it.  (With the second part cut
// off instead, twice that, of one sign for factors of like bits: 1 + 2^-8 - 2^-16 and the like 1.4e-7 off the 64-bit sum at K = 1,024
// instead of 0.7e-7.  The product of 777 rows, N 4,096, K 1,024 then takes 63.7 us instead of 65.4.)  Beyond bfloat16's range (and
// for what is no number) the third part is no number.
__device__ __forceinline__ void three_parts(float& x, float& y, uint32_t (&parts)[3]) {
    const __nv_bfloat162 first = __floats2bfloat162_rn(x, y);
    parts[0] = *reinterpret_cast<const uint32_t*>(&first);
    less_part(x, y, parts[0]);
    const __nv_bfloat162 second = __floats2bfloat162_rn(x, y);
    parts[1] = *reinterpret_cast<const uint32_t*>(&second);
    less_part(x, y, parts[1]);
    parts[2] = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
}
// Bits of a float32 that three parts leave: in what is left in place of the float (three_parts), the lower half is 0 unless bits of it lie
// under bfloat16's range (2^-133), or unless it is no number.
constexpr uint32_t LOST_BITS = 0xFFFF;
__device__ __forceinline__ uint32_t left_bits(float4 v) { return __float_as_uint(v.x) | __float_as_uint(v.y) | __float_as_uint(v.z) | __float_as_uint(v.w); }
