// Plain matrix product with a fused epilogue, float arithmetic only:
//   out[n, m] = act( sum_k a[n,k] * w[m,k] + bias[m] )       w stored [out, in]
// Every output element is one chain of fused multiply-adds over k in ascending
// order, whatever the number of rows, so a row's result does not depend on the
// batch it is in.  This is the matrix product of the 32-bit path (no tensor
// cores, no reduced-precision mode) and the plain twin of the bfloat16 one.
//
// The reference calls cuBLAS for all five products (src/csrc/util/cublas_wrapper.cc:29-53,
// call sites src/csrc/layer/attention.cc:102,255, src/csrc/layer/ffn.cc:71,96,
// src/csrc/model/gpt/gpt.cc:192) and adds bias / activation in separate kernels.
//
// Two kernels give that chain, with the same bits.  gemm_f32_kernel serves float operands whose rows are whole 16-byte
// pieces (k % 4 == 0, aligned); gemm_plain_kernel serves every other size and bfloat16 operands.
#include "common.cuh"

#define GBM 64
#define GBN 64
#define GBK 16

template <typename T, typename TO>
__global__ void __launch_bounds__(256)
gemm_plain_kernel(const T* __restrict__ a, const T* __restrict__ w, const float* __restrict__ bias,
                  TO* __restrict__ out, int n_rows, int n_out, int k_dim, int act) {
    __shared__ float sa[GBK][GBM + 4];
    __shared__ float sw[GBK][GBN + 4];
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;   // tx -> out features, ty -> rows
    const int row0 = blockIdx.y * GBM, col0 = blockIdx.x * GBN;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < k_dim; k0 += GBK) {
        // 64 x 16 elements of each operand, 256 threads -> 4 each
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const int idx = threadIdx.x + it * 256;
            const int r = idx / GBK, kk = idx % GBK;
            const int k = k0 + kk;
            const int ar = row0 + r, wr = col0 + r;
            sa[kk][r] = (ar < n_rows && k < k_dim) ? to_f32(a[(size_t)ar * k_dim + k]) : 0.f;
            sw[kk][r] = (wr < n_out && k < k_dim) ? to_f32(w[(size_t)wr * k_dim + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < GBK; ++kk) {
            float av[4], wv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) av[i] = sa[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) wv[j] = sw[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = row0 + ty * 4 + i;
        if (r >= n_rows) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = col0 + tx * 4 + j;
            if (c >= n_out) continue;
            float v = acc[i][j];
            if (bias) v += bias[c];
            out[(size_t)r * n_out + c] = from_f32<TO>(apply_act(v, act));
        }
    }
}

// ---- float operands in 16-byte pieces -------------------------------------------------------------------
// Rows of a and of w lie along k, so both are copied to shared memory as they stand ([row][BK] with four floats of
// padding per row) by 16-byte asynchronous copies, STAGES blocks of k deep, and read back four k at a time.  A warp's
// lanes are 4 rows x 8 outputs and a thread owns TM x TN outputs (rows 4 i + its row, outputs 8 j + its output).
__device__ __forceinline__ void gf_cp16(uint32_t dst, const float* src, int bytes) {     // bytes: 16, or 0 for zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}

template <int TM, int TN, int WR, int WC, int BK, int STAGES>
struct GemmF32 {
    static constexpr int BM = 4 * TM * WR, BN = 8 * TN * WC, THREADS = 32 * WR * WC, LD = BK + 4;
    static constexpr size_t SMEM = sizeof(float) * STAGES * (BM + BN) * LD;
};

// U: steps of four k whose operands are read together, while those of the U steps before are multiplied
template <int TM, int TN, int WR, int WC, int BK, int STAGES, int U, int BLOCKS>
__global__ void __launch_bounds__(32 * WR * WC, BLOCKS)
gemm_f32_kernel(const float* __restrict__ a, const float* __restrict__ w, const float* __restrict__ bias,
                float* __restrict__ out, int n_rows, int n_out, int k_dim, int act) {
    using S = GemmF32<TM, TN, WR, WC, BK, STAGES>;
    extern __shared__ __align__(16) float gf_smem[];
    constexpr int STAGE = (S::BM + S::BN) * S::LD;          // floats of a stage: rows of a, then rows of w
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row0 = blockIdx.y * S::BM, col0 = blockIdx.x * S::BN;
    // a thread copies the same 16-byte piece of every STEP-th row; rows past the end copy nothing (zeros) from a valid
    // address, and so does every row once k is through
    constexpr int PIECES = BK / 4, STEP = S::THREADS / PIECES;
    static_assert(S::THREADS % PIECES == 0 && PIECES % U == 0, "whole rows per pass of the block, whole groups per stage");
    constexpr int NA = (S::BM + STEP - 1) / STEP, NW = (S::BN + STEP - 1) / STEP;
    const int cr = threadIdx.x / PIECES, ck = (threadIdx.x % PIECES) * 4;
    const float *pa[NA], *pw[NW];
    int za[NA], zw[NW];
#pragma unroll
    for (int i = 0; i < NA; ++i) {
        const int r = row0 + cr + i * STEP;
        pa[i] = a + (size_t)min(r, n_rows - 1) * k_dim + ck;
        za[i] = r < n_rows ? 16 : 0;
    }
#pragma unroll
    for (int i = 0; i < NW; ++i) {
        const int r = col0 + cr + i * STEP;
        pw[i] = w + (size_t)min(r, n_out - 1) * k_dim + ck;
        zw[i] = r < n_out ? 16 : 0;
    }
    const uint32_t dst_a = (uint32_t)__cvta_generic_to_shared(gf_smem) + (uint32_t)(cr * S::LD + ck) * 4u;
    const uint32_t dst_w = dst_a + (uint32_t)(S::BM * S::LD) * 4u;
    int k_left = k_dim - ck;                                // at the stage that is copied next
    auto load = [&](int stage) {
        const uint32_t at = (uint32_t)(stage * STAGE) * 4u;
        const int on = k_left > 0 ? -1 : 0;
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            if (NA * STEP == S::BM || cr + i * STEP < S::BM)
                gf_cp16(dst_a + at + (uint32_t)(i * STEP * S::LD) * 4u, on ? pa[i] : a, za[i] & on);
            pa[i] += BK;
        }
#pragma unroll
        for (int i = 0; i < NW; ++i) {
            if (NW * STEP == S::BN || cr + i * STEP < S::BN)
                gf_cp16(dst_w + at + (uint32_t)(i * STEP * S::LD) * 4u, on ? pw[i] : w, zw[i] & on);
            pw[i] += BK;
        }
        k_left -= BK;
    };
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    // lanes l and l ^ 1 (for w) or l ^ 2 (for a) read the same 16 bytes: a read of the warp then takes two cycles of shared
    // memory and not four
    const int ar = (warp / WC) * 4 * TM + ((lane & 1) | ((lane >> 4) << 1));
    const int wr = (warp % WC) * 8 * TN + ((lane >> 1) & 7);
    const int n_k = (k_dim + BK - 1) / BK;
#pragma unroll
    for (int p = 0; p < STAGES - 1; ++p) {
        if (p < n_k) load(p);
        asm volatile("cp.async.commit_group;\n" ::);
    }
    int stage = 0, fill = STAGES - 1;
    for (int kt = 0; kt < n_k; ++kt) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2));
        __syncthreads();         // this stage has landed for every thread, and every thread is done with the one before
        if (kt + STAGES - 1 < n_k) load(fill);
        asm volatile("cp.async.commit_group;\n" ::);
        const float* sa = gf_smem + (size_t)stage * STAGE + ar * S::LD;
        const float* sw = gf_smem + (size_t)stage * STAGE + (S::BM + wr) * S::LD;
        float4 av[2][U][TM], wv[2][U][TN];
        auto fetch = [&](int g) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
#pragma unroll
                for (int i = 0; i < TM; ++i)
                    av[g & 1][u][i] = *reinterpret_cast<const float4*>(sa + 4 * i * S::LD + (g * U + u) * 4);
#pragma unroll
                for (int j = 0; j < TN; ++j)
                    wv[g & 1][u][j] = *reinterpret_cast<const float4*>(sw + 8 * j * S::LD + (g * U + u) * 4);
            }
        };
        fetch(0);
#pragma unroll
        for (int g = 0; g < PIECES / U; ++g) {
            if (g + 1 < PIECES / U) fetch(g + 1);
#pragma unroll
            for (int u = 0; u < U; ++u) {
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const float4 b = wv[g & 1][u][j];
#pragma unroll
                    for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(av[g & 1][u][i].x, b.x, acc[i][j]);
#pragma unroll
                    for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(av[g & 1][u][i].y, b.y, acc[i][j]);
#pragma unroll
                    for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(av[g & 1][u][i].z, b.z, acc[i][j]);
#pragma unroll
                    for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(av[g & 1][u][i].w, b.w, acc[i][j]);
                }
            }
        }
        if (++stage == STAGES) stage = 0;
        if (++fill == STAGES) fill = 0;
    }
#pragma unroll
    for (int j = 0; j < TN; ++j) {
        const int c = col0 + wr + 8 * j;
        if (c >= n_out) continue;
        const float b = bias ? bias[c] : 0.f;
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int r = row0 + ar + 4 * i;
            if (r >= n_rows) continue;
            out[(size_t)r * n_out + c] = apply_act(bias ? acc[i][j] + b : acc[i][j], act);
        }
    }
}

template <int TM, int TN, int WR, int WC, int BK, int STAGES, int U, int BLOCKS>
static int gemm_f32_launch(const float* a, const float* w, const float* bias, float* out, int n_rows, int n_out, int k_dim,
                           int act, cudaStream_t s) {
    using S = GemmF32<TM, TN, WR, WC, BK, STAGES>;
    auto kernel = gemm_f32_kernel<TM, TN, WR, WC, BK, STAGES, U, BLOCKS>;
    dim3 grid((n_out + S::BN - 1) / S::BN, (n_rows + S::BM - 1) / S::BM);
    if (grid.y > 65535) return ST_ERR_TOO_LARGE;
    if (S::SMEM > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
        if (e != cudaSuccess) return (int)e;
    }
    kernel<<<grid, S::THREADS, S::SMEM, s>>>(a, w, bias, out, n_rows, n_out, k_dim, act);
    return st_launch_status();
}

// Which tile.  Measured on one B200, times with the 6 us of an empty launch between events, L2 flushed; in brackets what the
// kernel of 64 x 64 tiles with 4 x 4 outputs per thread took, which served every size before.
//   up to 8 rows: bound by the weights' way from memory (and below that by the chain: four clocks per multiply-add, so
//     k = 4096 takes 8.4 us however the work is spread).  Tiles as narrow as the rows; 256 or 512 bytes of a row per stage
//     and eight or six stages keep 35 to 100 KB per block under way.  8 x 4096 x 4096 29.7 us, 67 MB (455); with 16 or 32
//     outputs per block, whichever gives the SMs a block each: 1 x 2048 x 2048 14 us with 16; and where there are three
//     halves of a block of 32 per SM two warps of 2 x 2 outputs pull more weights per instruction: 8 x 2048 x 8192 26.6 us
//     (30.8 with four warps of 2 x 1), 8 x 2048 x 50272 106 us = 4.1 TB/s (119)
//   up to 16 rows: one tile of 16 rows while it fills three quarters of the SMs (16 x 2048 x 8192: 32.8 us, 43 with two of 8)
//   prompts: bound by the multiply-adds (with three operands from registers 60 of the nominal 74 TFLOP/s, measured alone).
//     8 x 4 outputs per thread from four blocks of 64 x 64 per SM: 1000 x 2048 x 8192 775 us = 43 TFLOP/s (1490 us, 23);
//     8 x 8 outputs spill or leave two warps per scheduler (938 us).  Chains of even and odd k side by side in paired
//     multiply-adds gave 725 us and another order of the sum: not taken.  With about one 64 x 64 tile per SM its
//     256-thread form wins (128 x 4096 x 4096: 135 us, 146 with 32 x 32), and with fewer, or between one and four, 32 x 32
//     (600 x 2048 x 2048: 161 us, 176 with 64 x 64).
static int gemm_f32(const float* a, const float* w, const float* bias, float* out, int n_rows, int n_out, int k_dim, int act,
                    cudaStream_t s) {
    const int sms = st_sm_count();
    auto blocks = [&](int bm, int bn) { return (long long)((n_rows + bm - 1) / bm) * ((n_out + bn - 1) / bn); };
#define GF(...) return gemm_f32_launch<__VA_ARGS__>(a, w, bias, out, n_rows, n_out, k_dim, act, s)
    if (n_rows <= 4) {
        if (2 * blocks(4, 32) < sms) GF(1, 1, 1, 2, 64, 8, 4, 3);        // 4 x 16
        GF(1, 1, 1, 4, 64, 8, 4, 2);                                     // 4 x 32
    }
    if (n_rows <= 8) {
        if (2 * blocks(8, 32) > 3 * sms) GF(2, 2, 1, 2, 64, 8, 2, 2);    // 8 x 32, two warps
        if (4 * blocks(8, 32) > 3 * sms) GF(2, 1, 1, 4, 128, 6, 4, 1);   // 8 x 32, four warps
        GF(2, 1, 1, 2, 64, 8, 4, 3);                                     // 8 x 16
    }
    if (n_rows <= 16) {
        if (4 * blocks(16, 64) > 3 * sms) GF(4, 2, 1, 4, 64, 4, 2, 2);   // 16 x 64
        GF(2, 1, 1, 2, 64, 8, 4, 3);                                     // 8 x 16
    }
    if (blocks(64, 64) >= 4 * sms) GF(8, 4, 2, 2, 32, 3, 1, 4);          // 64 x 64, 8 x 4 outputs per thread
    if (4 * blocks(64, 64) > 3 * sms && blocks(64, 64) <= sms) GF(4, 4, 4, 2, 32, 3, 1, 2);     // 64 x 64, 4 x 4
    if (blocks(32, 32) <= sms) GF(4, 2, 2, 2, 64, 4, 2, 2);              // 32 x 32, 64 k per stage
    GF(4, 2, 2, 2, 32, 6, 2, 3);                                         // 32 x 32
#undef GF
}

ST_EXPORT int st_gemm_plain(const void* a, const void* w, const float* bias, void* out, int n_rows, int n_out,
                            int k_dim, int act, int dtype, int out_f32, void* stream) {
    if (n_rows <= 0 || n_out <= 0) return 0;
    if (k_dim <= 0) return ST_ERR_BAD_SIZE;
    cudaStream_t s = (cudaStream_t)stream;
    dim3 grid((n_out + GBN - 1) / GBN, (n_rows + GBM - 1) / GBM);
    if (grid.y > 65535) return ST_ERR_TOO_LARGE;
    if (dtype == 0 && k_dim % 4 == 0 && aligned16(a) && aligned16(w))
        return gemm_f32((const float*)a, (const float*)w, bias, (float*)out, n_rows, n_out, k_dim, act, s);
    if (dtype == 0)
        gemm_plain_kernel<float, float><<<grid, 256, 0, s>>>((const float*)a, (const float*)w, bias, (float*)out,
                                                              n_rows, n_out, k_dim, act);
    else if (dtype == 1) {
        if (out_f32)
            gemm_plain_kernel<bf16, float><<<grid, 256, 0, s>>>((const bf16*)a, (const bf16*)w, bias, (float*)out,
                                                                 n_rows, n_out, k_dim, act);
        else
            gemm_plain_kernel<bf16, bf16><<<grid, 256, 0, s>>>((const bf16*)a, (const bf16*)w, bias, (bf16*)out,
                                                                n_rows, n_out, k_dim, act);
    } else return ST_ERR_BAD_DTYPE;
    return st_launch_status();
}
