// A float as the sum of three bfloat16 numbers of eight bits each: x = h + m + l, h = bf16(x), m = bf16(x - h), l = bf16(x - h - m),
// each difference exact.  Products of such parts are exact in the tensor cores' float accumulator (gemm_f32.cuh says which of them
// are formed, in which order, and what they leave out).
#pragma once
#include "common.cuh"

// what two bfloat16 numbers leave of two floats
__device__ __forceinline__ void gf_rest(float& x0, float& x1, uint32_t packed) {
    asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %3};\n\tsub.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}\n"
        : "+f"(x0), "+f"(x1) : "f"(__uint_as_float(packed << 16)), "f"(__uint_as_float(packed & 0xffff0000u)));
}
// two neighbours -> their three parts, packed
__device__ __forceinline__ void gf_split(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
    const __nv_bfloat162 hb = __floats2bfloat162_rn(x0, x1);
    h = *reinterpret_cast<const uint32_t*>(&hb);
    gf_rest(x0, x1, h);
    const __nv_bfloat162 mb = __floats2bfloat162_rn(x0, x1);
    m = *reinterpret_cast<const uint32_t*>(&mb);
    gf_rest(x0, x1, m);
    const __nv_bfloat162 lb = __floats2bfloat162_rn(x0, x1);
    l = *reinterpret_cast<const uint32_t*>(&lb);
}
