// A float, scaled up by 2^16, as the sum of three bfloat16 numbers of eight bits each: 2^16 x = h + m + l, h = bf16(2^16 x),
// m = bf16(2^16 x - h), l = bf16(2^16 x - h - m), each difference exact.  Unscaled, the last bits of floats below 2^-110 would fall under the
// smallest bfloat16 (2^-133): numbers of 2^-120 came out of a product off by 3.5e-5 of themselves.  So every float below 2^112 is held
// to its last bit; above that h is infinite, and sums that are not finite are formed again from the floats.  Products of such parts
// are exact in the tensor cores' float accumulator (gemm_f32.cuh says which of them are formed, in which order, and what they
// leave out).  A number cut into slices whose products are exact: T. J. Dekker, "A floating-point technique for extending the available
// precision", Numerische Mathematik 18 (1971).
#pragma once
#include "common.cuh"

#define GF_UP 65536.f                      // a float's scale
#define GF_DOWN 1.52587890625e-5f          // and back: a sum of products of one split operand with another that is not
#define GF_DOWN2 2.3283064365386963e-10f   // of two split operands

// what two bfloat16 numbers leave of two floats
__device__ __forceinline__ void gf_rest(float& x0, float& x1, uint32_t packed) {
    asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %3};\n\tsub.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}\n"
        : "+f"(x0), "+f"(x1) : "f"(__uint_as_float(packed << 16)), "f"(__uint_as_float(packed & 0xffff0000u)));
}
// two neighbours -> their three parts, packed
__device__ __forceinline__ void gf_split(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
    asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %2};\n\tmul.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a;\n\t}\n"
        : "+f"(x0), "+f"(x1) : "f"(GF_UP));
    const __nv_bfloat162 hb = __floats2bfloat162_rn(x0, x1);
    h = *reinterpret_cast<const uint32_t*>(&hb);
    gf_rest(x0, x1, h);
    const __nv_bfloat162 mb = __floats2bfloat162_rn(x0, x1);
    m = *reinterpret_cast<const uint32_t*>(&mb);
    gf_rest(x0, x1, m);
    const __nv_bfloat162 lb = __floats2bfloat162_rn(x0, x1);
    l = *reinterpret_cast<const uint32_t*>(&lb);
}
// the float whose parts these are (h finite)
__device__ __forceinline__ float gf_join(float h, float m, float l) { return ((h + m) + l) * GF_DOWN; }
