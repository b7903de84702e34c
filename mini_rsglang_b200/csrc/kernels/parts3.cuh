// A float32 as three bfloat16: 8 + 8 + 8 bits of its significand, exact down to where the last part falls under bfloat16's range.
#pragma once
#include "common.cuh"

// x += y, two floats of a register pair at a time
__device__ __forceinline__ void add_pair(float& x0, float& x1, float y0, float y1) {
    asm("{\n .reg .b64 a, b;\n mov.b64 a, {%0, %1};\n mov.b64 b, {%2, %3};\n add.rn.f32x2 a, a, b;\n mov.b64 {%0, %1}, a;\n}" : "+f"(x0), "+f"(x1) : "f"(y0), "f"(y1));
}
// The next part of two floats as a pair of bfloat16; what the rounding leaves stays in them, exact.  Beyond bfloat16's range a part is
// infinite and what is left no number.
__device__ __forceinline__ uint32_t take_part(float& x, float& y) {
    const __nv_bfloat162 pair = __floats2bfloat162_rn(x, y);
    const uint32_t bits = *reinterpret_cast<const uint32_t*>(&pair);
    // x - part in one instruction, the part as it lies: no shift and no mask
    asm("{\n .reg .b16 lo, hi, minus;\n mov.b32 {lo, hi}, %2;\n mov.b16 minus, 0xBF80;\n fma.rn.f32.bf16 %0, lo, minus, %0;\n fma.rn.f32.bf16 %1, hi, minus, %1;\n}"
        : "+f"(x), "+f"(y) : "r"(bits));
    return bits;
}
