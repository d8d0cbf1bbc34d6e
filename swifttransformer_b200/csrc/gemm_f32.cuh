// The 32-bit matrix product on the tensor cores, out[n, m] = act( sum_k a[n,k] * w[m,k] + bias[m] ) with float operands and
// w stored [out, in]: what its kernels (gemm_f32_tc.cu for many rows, gemm_f32_few.cu for few) share.
//
// A float, times 2^16, is the sum of three bfloat16 numbers of eight bits each, h + m + l (float_parts.cuh); an output is the sum of their
// products times 2^-32.  Of the nine products of two such sums six are formed,
//   w_l a_h + w_h a_l + w_m a_m + w_m a_h + w_h a_m + w_h a_h,
// each exact in the tensor cores' float accumulator; the three left out are at most 2^-24 of w a together (on average 2^-28).  The
// tensor cores cut a sum off where a float addition rounds it (measured: 6e-8 of bias after four steps of 16 k, 1.2e-7 after eight), so a
// sum stays there for one group of 64 k only, the small products first: its 24 steps end with the four of w_h a_h.  The groups' sums are
// added up in float registers in ascending order, each addition rounded to nearest.  An output so depends on its own row of a and of w
// alone, and its bits are the same for every number of rows, tile and kernel: all form the same groups and add them in the same order
// (mma.sync and tcgen05.mma give the same bits for the same sixteen products; a test holds the kernels to it).
//
// A sum that comes out infinite or not a number (operands that are, operands from 2^112 on, outputs from 2^96 on) is formed again as
// a chain of fused multiply-adds over k, which is what such operands give in plain float.
//
// Error against 64 bits, relative 2-norm, normal operands of any size from 2^-135 on: k = 16 4.7e-8, 64 7.7e-8, 512 9.6e-8, 2048 1.3e-7,
// 8192 2.2e-7 (a chain of fused multiply-adds over k: 7.4e-8, 1.4e-7, 4.0e-7, 8.1e-7, 1.6e-6).
#pragma once
#include "common.cuh"
#include "float_parts.cuh"

#define GF_BK 64             // k of a group

struct GemmF32 {
    const float *a, *w, *bias;
    float* out;
    int n_rows, n_out, k_dim, act;
};
__device__ __forceinline__ float gf_finish(const GemmF32& p, float v, float bias) { return apply_act(p.bias ? v + bias : v, p.act); }

// gemm_f32_few.cu: chains of multiply-adds, for k below GF_SHORT.  The tensor cores cut a sum off, so a product of one k is off by 4.6e-8 of
// itself where a float multiplication is by 2.6e-8; k = 2 4.6e-8 (chain 3.0e-8), 4 4.7e-8 (4.0e-8), 8 4.8e-8 (5.3e-8; of positive numbers 4.8e-8 and
// 4.6e-8), 16 4.7e-8 (7.4e-8).
#define GF_SHORT 9
int gf_short_launch(const GemmF32& p, cudaStream_t s);

// the same file: in tiles of 8 or 16 rows, and about what it takes, in units of 10 ns, with the form (-8, -16) that takes less
int gf_few_launch(const GemmF32& p, int rows, cudaStream_t s);
long long gf_few_cost(const GemmF32& p, int& form);
