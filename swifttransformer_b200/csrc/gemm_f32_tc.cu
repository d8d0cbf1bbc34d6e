// The 32-bit matrix product for more than a few rows on the 5th-generation tensor cores: see gemm_f32.cuh for the arithmetic.
//
// gemm_f32_split_kernel writes the three parts of a side by side, [3][n_rows][k rounded up to 64] bfloat16.  Then a block holds 128
// rows of w (the lanes of tensor memory) and nt <= 128 rows of a, and walks through k in groups of 64:
//   warp 8      copies w by TMA (boxes of 128 rows x 32 floats, 128-byte swizzle) through a ring of stages
//   warp 9      issues the products
//   warp 10     copies the parts of a, one box of [3][nt][64] per group
//   warps 12-   split w, a thread per row: three parts into tensor memory, the A operand.  SETS times four warps, each set every
//               SETS-th group (a set takes about 2300 clocks for one; the products of one 12 nt)
//   warps 0-7   add a group's sums to their registers (half of the columns each, two to an instruction: 178.5 us among other passes for
//               1000 x 2048 x 8192, one by one 181.6) and store the results
// Both operands have two or (nt <= 64) four buffers, the sums two.  A group's products wait once, on a barrier that counts its
// parts of w, its box of a and the reading of the sums two groups before: with a wait for each the tensor cores stood still for 1000
// clocks of 2500 per group, for their queue is shorter than that.
// w in tensor memory and not in shared: a product then reads 4 KB of shared memory in its 64 clocks and not 8, and its rate is that
// of the tensor cores for any nt.  w is split by each block that uses it, for w is the larger operand and read from memory once.
//
// Bound by the tensor cores (24 products of 12 nt clocks a group; nt 128: 1670 clocks a group measured, 1536 of them products) and the
// power limit for prompts, by the chain split - products - sum of a group for few rows.  us on one B200, recorded calls over weights that
// are not in cache, in brackets the float multiply-adds that served before: 1000 x 2048 x 8192 149 (766; 176 in a run of other work, whose
// power holds the clock down), 1000 x 8192 x 2048 151 (923), 1000 x 4096 x 4096 148 (773), 128 x 2048 x 8192 32 (123), 64 x 8192 x 2048 74 (92),
// 33 x 2048 x 2048 22.5 (25.5), 64 x 768 x 2304 12.1 (12.1).
//
// Waits are bounded: one that expires marks the block dead, `status` gets 5, and the block waits (again with a limit) for its
// copies under way, frees its tensor memory and leaves.
#include "gemm_f32.cuh"
#include "tcgen05.cuh"
#include "tma_host.h"

#define GF_BM 128
#define GF_SETS(NT) ((NT) <= 64 ? 4 : 2)
#define GF_THREADS(NT) (384 + 128 * GF_SETS(NT))
#define GF_STAGE (GF_BM * GF_BK * 4u)        // bytes of w per stage: two boxes of [128][32] floats
#define GF_MAX_STAGES 6
#define GF_MAX_BUFS 4
#define GF_SMEM (225 * 1024)

struct GemmF32Tc {
    GemmF32 g;
    int nt, n_tiles, tiles;          // rows of a per tile (a multiple of 16), tiles of rows, tiles in all
    int stages, vec_w;
};

__device__ __forceinline__ void gf_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void gf_st8(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};\n"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void gf_ld8(uint32_t taddr, float* v) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr) : "memory");
}

// a thread per eight neighbours of a row
__global__ void __launch_bounds__(256)
gemm_f32_split_kernel(const float* __restrict__ a, uint4* __restrict__ parts, int n_rows, int k_dim, int k_pad, int vec) {
    ST_PDL_TRIGGER();
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x, per_row = k_pad / 8, n = (size_t)n_rows * per_row;
    if (i >= n) return;
    const int row = (int)(i / per_row), k = (int)(i % per_row) * 8;
    const float* src = a + (size_t)row * k_dim + k;
    float v[8];
    if (vec) {
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 x = k < k_dim ? __ldcg(reinterpret_cast<const float4*>(src)) : z;
        const float4 y = k + 4 < k_dim ? __ldcg(reinterpret_cast<const float4*>(src + 4)) : z;
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = k + j < k_dim ? __ldcg(src + j) : 0.f;
    }
    uint32_t h[4], m[4], l[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) gf_split(v[2 * j], v[2 * j + 1], h[j], m[j], l[j]);
    parts[i] = make_uint4(h[0], h[1], h[2], h[3]);
    parts[n + i] = make_uint4(m[0], m[1], m[2], m[3]);
    parts[2 * n + i] = make_uint4(l[0], l[1], l[2], l[3]);
}

// Outputs that came out infinite or not a number, again as chains of multiply-adds over k: all threads of a block walk through its tiles
// once the pipeline has ended, where no warp waits for them under a limit, and multiply every tile that has such an output (128
// x nt sums side by side, 32 k at a time through the pipeline's shared memory) until all of its sums of interest are no numbers, or
// to the end.  us for 1000 x 2048 x 8192: 166 where all are finite, 1064 with one infinity among the operands, 3513 with one in every row.
template <int NT>
__device__ __noinline__ void gf_chains(const GemmF32Tc& p, float* smem) {
    constexpr int NR = NT / 16, LD = 33;
    const GemmF32& q = p.g;
    float *W = smem, *A = smem + GF_BM * LD;                  // [128][33], [nt][33]
    const int tid = threadIdx.x, cl = tid & 31, rl = tid >> 5;
    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
        const int m0 = tile / p.n_tiles * GF_BM, n0 = tile % p.n_tiles * p.nt;
        // 512 threads: columns cl + 32 i, rows rl + 16 j; wanted: bit 4 j + i
        auto out_at = [&](int i, int j) { return q.out + (size_t)(n0 + rl + 16 * j) * q.n_out + m0 + cl + 32 * i; };
        uint32_t wanted = 0;
#pragma unroll 1
        for (int x = 0; x < 4 * NR; ++x) {
            const int i = x & 3, j = x >> 2;
            if (rl < 16 && 16 * j < p.nt && n0 + rl + 16 * j < q.n_rows && m0 + cl + 32 * i < q.n_out && !(fabsf(*out_at(i, j)) < INFINITY))
                wanted |= 1u << x;
        }
        if (!__syncthreads_or(wanted != 0)) continue;
        float s[NR][4] = {};
#pragma unroll 1
        for (int k0 = 0; k0 < q.k_dim; k0 += 32) {
            bool open = false;
#pragma unroll
            for (int x = 0; x < 4 * NR; ++x) open |= (wanted >> x & 1) && s[x >> 2][x & 3] == s[x >> 2][x & 3];
            if (!__syncthreads_or(open)) break;
            for (int i = rl; i < GF_BM + p.nt; i += blockDim.x / 32) {
                const bool is_w = i < GF_BM;
                const int row = is_w ? m0 + i : n0 + i - GF_BM, k = k0 + cl;
                smem[i * LD + cl] = row < (is_w ? q.n_out : q.n_rows) && k < q.k_dim ? __ldg((is_w ? q.w : q.a) + (size_t)row * q.k_dim + k) : 0.f;
            }
            __syncthreads();
            if (rl < 16)
#pragma unroll 4
                for (int k = 0; k < 32; ++k) {
                    float w[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) w[i] = W[(cl + 32 * i) * LD + k];
#pragma unroll
                    for (int j = 0; j < NR; ++j) {
                        if (16 * j >= p.nt) break;
                        const float a = A[(rl + 16 * j) * LD + k];
#pragma unroll
                        for (int i = 0; i < 4; ++i) s[j][i] = fmaf(a, w[i], s[j][i]);
                    }
                }
        }
#pragma unroll
        for (int x = 0; x < 4 * NR; ++x)
            if (wanted >> x & 1) *out_at(x & 3, x >> 2) = gf_finish(q, s[x >> 2][x & 3], q.bias ? __ldg(q.bias + m0 + cl + 32 * (x & 3)) : 0.f);
    }
}

template <int NT>
__global__ void __launch_bounds__(GF_THREADS(NT), 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap a_map,
                   const __grid_constant__ GemmF32Tc p, int* status) {
    extern __shared__ unsigned char gf_raw[];
    // w landed / read; a group's operands in place and its sums' place free; its products complete
    __shared__ __align__(8) unsigned long long s_wfull[GF_MAX_STAGES], s_wfree[GF_MAX_STAGES], s_ready[GF_MAX_BUFS], s_done[GF_MAX_BUFS];
    __shared__ uint32_t s_tmem;
    __shared__ int s_dead, s_issued, s_odd;
    constexpr int BUFS = NT <= 64 ? 4 : 2;                   // a power of two
    constexpr int W_COL = NT <= 64 ? 128 : 256;              // tensor memory: sums at 0 and W_COL / 2, parts of w from W_COL on, 96 each
    const GemmF32& q = p.g;
    const uint32_t part = p.nt * 128u, a_stage = 3 * part;   // bytes of one part of a group of a ([nt][64]: multiples of 1024)
    const uint32_t base = (tc_smem(gf_raw) + 1023u) & ~1023u;
    const uint32_t sA = base, sW = base + BUFS * a_stage;
    const int tid = threadIdx.x, warp = tc_warp(), lane = tid & 31;
    volatile int* dead = &s_dead;
    if (tid == 0) {
        for (int s = 0; s < GF_MAX_STAGES; ++s) { tc_mbar_init(tc_smem(&s_wfull[s]), 1); tc_mbar_init(tc_smem(&s_wfree[s]), 4); }
        for (int i = 0; i < BUFS; ++i) {
            tc_mbar_init(tc_smem(&s_ready[i]), 13);          // four warps of w's parts, the copy of a, eight warps that read sums
            tc_mbar_init(tc_smem(&s_done[i]), 1);
        }
        tc_mbar_init_fence();
        s_dead = 0;
        s_issued = 0;
        s_odd = 0;
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem(&s_tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = s_tmem;
    const int n_groups = (q.k_dim + GF_BK - 1) / GF_BK;
    const int first = blockIdx.x, step = gridDim.x;
    auto m_of = [&](int tile) { return tile / p.n_tiles * GF_BM; };          // tiles of one part of w side by side
    auto n_of = [&](int tile) { return tile % p.n_tiles * p.nt; };

    if (warp == 8) {
        // ---- copies of w
        if (p.vec_w) {
            int it = 0, s = 0, turn = 0;
            bool ok = true;
            for (int tile = first; ok && tile < p.tiles; tile += step) {
                const int m0 = m_of(tile);
                for (int g = 0; g < n_groups; ++g) {
                    if (turn > 0) ok = tc_wait_warp(tc_smem(&s_wfree[s]), (turn - 1) & 1, dead);
                    if (!ok) break;
                    const uint32_t mb = tc_smem(&s_wfull[s]), dst = sW + s * GF_STAGE;
                    ++it;
                    if (tc_elect()) {
                        tc_mbar_expect_tx(mb, GF_STAGE);
                        tc_tma_load_2d(dst, &w_map, g * GF_BK, m0, mb);
                        tc_tma_load_2d(dst + GF_STAGE / 2, &w_map, g * GF_BK + 32, m0, mb);
                        s_issued = it;
                    }
                    __syncwarp();
                    if (++s == p.stages) { s = 0; ++turn; }
                }
            }
        }
    } else if (warp == 10) {
        // ---- copies of a's parts, which the kernel before wrote
        ST_PDL_WAIT();
        int it = 0;
        bool ok = true;
        for (int tile = first; ok && tile < p.tiles; tile += step) {
            const int n0 = n_of(tile);
            for (int g = 0; g < n_groups; ++g, ++it) {
                const int buf = it % BUFS;
                if (it >= BUFS) ok = tc_wait_warp(tc_smem(&s_done[buf]), (it / BUFS - 1) & 1, dead);
                if (!ok) break;
                const uint32_t mb = tc_smem(&s_ready[buf]);
                if (tc_elect()) {
                    tc_mbar_expect_tx(mb, a_stage);
                    tc_tma_load_3d(sA + buf * a_stage, &a_map, g * GF_BK, n0, 0, mb);
                }
                __syncwarp();
            }
        }
    } else if (warp == 9) {
        // ---- products
        const uint32_t idesc = tc_idesc(GF_BM, p.nt, 0, 0);
        int it = 0;
        bool ok = true;
        for (int tile = first; ok && tile < p.tiles; tile += step)
            for (int g = 0; g < n_groups; ++g, ++it) {
                const int buf = it % BUFS;
                ok = tc_wait_warp(tc_smem(&s_ready[buf]), (it / BUFS) & 1, dead);
                if (!ok) break;
                tc_fence_after_sync();
                const uint32_t d = tmem + (it & 1) * (W_COL / 2), wa = tmem + W_COL + buf * 96;
                const uint64_t da = tc_desc(sA + buf * a_stage, 16, 1024);
                constexpr int W_PART[6] = {2, 0, 1, 1, 0, 0}, A_PART[6] = {0, 2, 1, 0, 1, 0};
                if (tc_elect()) {
#pragma unroll
                    for (int x = 0; x < 6; ++x)
#pragma unroll
                        for (int kk = 0; kk < GF_BK / 16; ++kk)
                            tc_mma_ts(d, wa + W_PART[x] * 32 + kk * 8, da + ((A_PART[x] * part + kk * 32) >> 4), idesc, x > 0 || kk > 0);
                    tc_commit(tc_smem(&s_done[buf]));
                }
                __syncwarp();
            }
    } else if (warp >= 12) {
        // ---- rows of w: a thread splits 64 neighbours of one row, its lane of tensor memory
        constexpr int SETS = GF_SETS(NT);
        const int mine = (warp - 12) >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + W_COL;
        int it = 0, s = 0, turn = 0;
        bool ok = true;
        for (int tile = first; ok && tile < p.tiles; tile += step) {
            const int m = m_of(tile) + row;
            for (int g = 0; g < n_groups; ++g, ++it) {
                if (it % SETS == mine) {
                    const int buf = it % BUFS;
                    // The products that read this buffer last are complete.  This wait comes first: behind it every earlier stage
                    // has landed (there are at least as many stages as buffers), and the next one is asked for the phase that
                    // follows; before it a copy of two turns ago may still be under way, whose phase has the same parity.
                    if (it >= BUFS) ok = tc_wait_warp(tc_smem(&s_done[buf]), (it / BUFS - 1) & 1, dead);
                    if (ok && p.vec_w) ok = tc_wait_warp(tc_smem(&s_wfull[s]), turn & 1, dead);
                    if (!ok) break;
                    tc_fence_after_sync();
#pragma unroll 2
                    for (int c = 0; c < 4; ++c) {            // sixteen at a time
                        float f[16];
                        if (p.vec_w) {
                            const uint32_t src = sW + s * GF_STAGE + (c >> 1) * (GF_STAGE / 2) + row * 128;
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];\n"
                                             : "=f"(f[4 * e]), "=f"(f[4 * e + 1]), "=f"(f[4 * e + 2]), "=f"(f[4 * e + 3])
                                             : "r"(src + ((((c & 1) * 4 + e) ^ (row & 7)) << 4)));
                        } else {
                            const int k = g * GF_BK + c * 16;
                            const float* src = q.w + (size_t)min(m, q.n_out - 1) * q.k_dim + k;
#pragma unroll
                            for (int e = 0; e < 16; ++e) f[e] = m < q.n_out && k + e < q.k_dim ? __ldg(src + e) : 0.f;
                        }
                        uint32_t h[8], md[8], l[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) gf_split(f[2 * e], f[2 * e + 1], h[e], md[e], l[e]);
                        const uint32_t dst = at + buf * 96 + c * 8;
                        gf_st8(dst, h);
                        gf_st8(dst + 32, md);
                        gf_st8(dst + 64, l);
                    }
                    tc_st_wait();
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) {
                        gf_arrive(tc_smem(&s_ready[buf]));
                        if (p.vec_w) gf_arrive(tc_smem(&s_wfree[s]));
                    }
                }
                if (++s == p.stages) { s = 0; ++turn; }
            }
        }
    } else if (warp < 8) {
        // ---- sums
        const int quarter = warp & 3, half = warp >> 2, cols = p.nt / 2;          // this warp's columns: half * cols ..
        const uint32_t src = tmem + ((uint32_t)(quarter * 32) << 16) + half * cols;
        int it = 0;
        bool ok = true;
        if (lane == 0) {                                                          // the first two groups' places are free
            gf_arrive(tc_smem(&s_ready[0]));
            gf_arrive(tc_smem(&s_ready[1]));
        }
        for (int tile = first; ok && tile < p.tiles; tile += step) {
            const int col = m_of(tile) + quarter * 32 + lane, n0 = n_of(tile) + half * cols;
            const int live = min(cols, q.n_rows - n0);                            // may be negative
            float acc[NT / 2];
#pragma unroll
            for (int j = 0; j < NT / 2; ++j) acc[j] = 0.f;
            for (int g = 0; g < n_groups; ++g, ++it) {
                ok = tc_wait_warp(tc_smem(&s_done[it % BUFS]), (it / BUFS) & 1, dead);
                if (!ok) break;
                tc_fence_after_sync();
#pragma unroll
                for (int j = 0; j < NT / 2; j += 16) {
                    float v[16];
#pragma unroll
                    for (int e = 0; e < 16; e += 8)
                        if (j + e < cols) gf_ld8(src + (it & 1) * (W_COL / 2) + j + e, v + e);
                    tc_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; e += 2)
                        if (j + (e & 8) < cols) tc_add2(acc[j + e], acc[j + e + 1], v[e], v[e + 1]);
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) gf_arrive(tc_smem(&s_ready[(it + 2) % BUFS]));
            }
            if (ok && col < q.n_out) {
                // The registers are stored by unrolled code, which has to be short: with every activation in it 20 us of a tile's
                // 48 went into fetching instructions.  What is not short is done to the stored sums, one after the other; those that
                // are not finite stay as they are for gf_chains.
                const float bias = q.bias ? __ldg(q.bias + col) : 0.f;
                float* dst = q.out + (size_t)n0 * q.n_out + col;
                bool odd = false;
#pragma unroll
                for (int j = 0; j < NT / 2; ++j) odd |= j < live && !(fabsf(acc[j]) < INFINITY);
                const bool later = odd || q.act > 1;
#pragma unroll
                for (int j = 0; j < NT / 2; ++j)
                    if (j < live) {
                        float v = acc[j] * GF_DOWN2;
                        if (!later && q.bias) v += bias;
                        if (!later && q.act == 1) v = v > 0.f ? v : 0.f;
                        dst[(size_t)j * q.n_out] = v;
                    }
                if (odd) s_odd = 1;
                if (later)
#pragma unroll 1
                    for (int j = 0; j < live; ++j) {
                        const float v = dst[(size_t)j * q.n_out];
                        if (fabsf(v) < INFINITY) dst[(size_t)j * q.n_out] = gf_finish(q, v, bias);
                    }
            }
            __syncwarp();
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (s_dead && tid == 0) {
        // copies and products under way end before the block's memory is given up: a stage of w by its barrier, a's boxes and the
        // products by time, a few milliseconds
        if (status) atomicExch(status, 5);
        for (int s = 0; s < p.stages && s < s_issued; ++s) tc_wait(tc_smem(&s_wfull[s]), ((s_issued - 1 - s) / p.stages) & 1);
        for (int i = 0; i < 20000; ++i) __nanosleep(100);
    }
    __syncthreads();
    if (s_odd && !s_dead) gf_chains<NT>(p, reinterpret_cast<float*>(gf_raw));
    if (warp == 9) {
        tc_fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512) : "memory");
    }
}

template <int NT>
static int gf_launch(const CUtensorMap& w_map, const CUtensorMap& a_map, const GemmF32Tc& p, int grid, int* status, cudaStream_t s) {
    auto kernel = gemm_f32_tc_kernel<NT>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GF_SMEM);
    if (e != cudaSuccess) return (int)e;
    return st_launch_pdl("gemm_f32", kernel, dim3((unsigned)grid), dim3(GF_THREADS(NT)), GF_SMEM, s, w_map, a_map, p, status);
}

// The form (see st_gemm_f32) by what they were measured to take (units of 10 ns, on one B200, recorded calls): a tile's group
// 46 + nt / 3 up to 64 rows, 50 + nt / 2 above (two sets of splitting warps and two buffers then), a round of tiles 200 beside that and
// the splitting kernel and the launch 450; twelve times as much for the groups but two where rows of w are not whole pieces of 16 bytes
// (40 x 770 x 2304 87 us, 40 x 130 x 512 10).  us, this kernel / gemm_f32_few.cu: 16 x 768 x 3072 12.1 / 8.4, 16 x 2048 x 6144 23.5 / 27.6,
// 24 x 4096 x 4096 40.2 / 52.8, 24 x 8192 x 2048 73 / 55, 1 x 768 x 50272 35 / 41, 64 x 64 x 64 5.7 / 3.5.
#define GF_FORM_SHORT 1
static int gf_plan(const GemmF32& g) {
    if (g.k_dim < GF_SHORT) return GF_FORM_SHORT;
    const long long sms = st_sm_count(), m_tiles = ((long long)g.n_out + GF_BM - 1) / GF_BM, n_groups = ((long long)g.k_dim + GF_BK - 1) / GF_BK;
    const int rows16 = g.n_rows >= 128 ? 128 : (g.n_rows + 15) / 16 * 16;
    int form;
    long long best = gf_few_cost(g, form);
    for (int t = 16; t <= rows16; t += 16) {
        const long long tiles = m_tiles * (((long long)g.n_rows + t - 1) / t);
        const long long groups = g.k_dim % 4 == 0 || n_groups <= 2 ? n_groups : 12 * (n_groups - 2);
        const long long cost = 450 + (tiles + sms - 1) / sms * (groups * (t <= 64 ? 46 + t / 3 : 50 + t / 2) + 200);
        if (cost < best) { best = cost; form = t; }
    }
    return form;
}

static long long gf_row_bytes(int k_dim) { return 6 * (((long long)k_dim + GF_BK - 1) / GF_BK * GF_BK); }

// Bytes of scratch with which st_gemm_f32 takes all rows at once on the current device, or, where that is more than `most`, as many rows as
// that holds in whole tiles of 128 at a time, at least one tile.  form: the one st_gemm_f32 chooses, so that a caller who keeps it by
// size saves each call the choice.
ST_EXPORT long long st_gemm_f32_scratch(int n_rows, int n_out, int k_dim, long long most, int* form) {
    const GemmF32 g = {nullptr, nullptr, nullptr, nullptr, n_rows, n_out, k_dim, 0};
    *form = 0;
    if (n_rows <= 0 || n_out <= 0 || k_dim <= 0) return 0;
    *form = gf_plan(g);
    if (*form < 16) return 0;
    const long long per_row = gf_row_bytes(k_dim), tiles = most / (per_row * 128), rows = 128 * (tiles > 1 ? tiles : 1);
    return per_row * (rows < n_rows ? rows : n_rows);
}

static int gf_run(const GemmF32& g, int nt, void* scratch, int* status, cudaStream_t s);

// a [n_rows, k_dim], w [n_out, k_dim], out [n_rows, n_out], float and contiguous, of any alignment.  scratch: 16-byte aligned, with status;
// both may be null where st_gemm_f32_scratch is 0; with fewer bytes than all rows take the rows go in parts.  form: rows of a per tile of
// this kernel (a multiple of 16 up to 128), -8 and -16: gemm_f32_few.cu in such tiles, 1: chains (k below GF_SHORT), 0: chosen here.
ST_EXPORT int st_gemm_f32(const float* a, const float* w, const float* bias, float* out, int n_rows, int n_out, int k_dim, int act,
                          int form, void* scratch, long long scratch_bytes, int* status, void* stream) {
    if (n_rows <= 0 || n_out <= 0) return 0;
    if (k_dim <= 0) return ST_ERR_BAD_SIZE;
    const GemmF32 g = {a, w, bias, out, n_rows, n_out, k_dim, act};
    cudaStream_t s = (cudaStream_t)stream;
    const int nt = form == 0 ? gf_plan(g) : form;
    if (nt == GF_FORM_SHORT) return k_dim < GF_SHORT ? gf_short_launch(g, s) : ST_ERR_BAD_ARG;
    if (nt == -8 || nt == -16) return gf_few_launch(g, -nt, s);
    if (!status || !scratch || !aligned16(scratch) || nt < 16 || nt > 128 || nt % 16) return ST_ERR_BAD_ARG;
    long long rows = scratch_bytes / gf_row_bytes(k_dim);
    if (rows >= n_rows) return gf_run(g, nt, scratch, status, s);
    if (rows >= nt) rows = rows / nt * nt;
    if (rows < 1) return ST_ERR_BAD_ARG;
    for (long long r0 = 0; r0 < n_rows; r0 += rows) {                // (a part's splitting kernel starts when the part before is done)
        GemmF32 part = g;
        part.a += r0 * k_dim;
        part.out += r0 * n_out;
        part.n_rows = (int)(n_rows - r0 < rows ? n_rows - r0 : rows);
        const int rc = gf_run(part, nt, scratch, status, s);
        if (rc) return rc;
    }
    return 0;
}

static int gf_run(const GemmF32& g, int nt, void* scratch, int* status, cudaStream_t s) {
    const int sms = st_sm_count(), n_rows = g.n_rows, n_out = g.n_out, k_dim = g.k_dim;
    const float *a = g.a, *w = g.w;
    const long long m_tiles = ((long long)n_out + GF_BM - 1) / GF_BM, n_groups = ((long long)k_dim + GF_BK - 1) / GF_BK;
    const long long k_pad = n_groups * GF_BK;
    GemmF32Tc p;
    p.g = g;
    p.vec_w = k_dim % 4 == 0 && aligned16(w);
    p.nt = nt;
    const long long n_tiles = ((long long)n_rows + nt - 1) / nt, tiles = m_tiles * n_tiles;
    if (tiles > 0x3fffffffLL || k_pad > 0x7fffffffLL) return ST_ERR_TOO_LARGE;
    p.n_tiles = (int)n_tiles; p.tiles = (int)tiles;
    const int stages = (GF_SMEM - 1024 - (nt <= 64 ? 4 : 2) * nt * 384) / (int)GF_STAGE;
    p.stages = stages > GF_MAX_STAGES ? GF_MAX_STAGES : stages;             // 4 to 6: at least as many as buffers
    CUtensorMap w_map = {}, a_map;
    st_tma_encode_fn enc = st_tma_encoder();
    if (!enc) return ST_ERR_BAD_ARG;
    if (p.vec_w) {
        const cuuint64_t d[2] = {(cuuint64_t)k_dim, (cuuint64_t)n_out}, st[1] = {(cuuint64_t)k_dim * 4};
        const cuuint32_t b[2] = {32, GF_BM}, el[2] = {1, 1};
        if (enc(&w_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(w), d, st, b, el, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            p.vec_w = 0;                                     // sizes no tensor map takes: plain loads
    }
    const unsigned long long ad[3] = {(unsigned long long)k_pad, (unsigned long long)n_rows, 3};
    const unsigned ab[3] = {64, (unsigned)nt, 3};
    if (st_tma_encode_bf16(&a_map, scratch, 3, ad, ab)) return ST_ERR_BAD_ARG;
    const long long pieces = (long long)n_rows * (k_pad / 8);
    if ((pieces + 255) / 256 > 0x7fffffffLL) return ST_ERR_TOO_LARGE;
    gemm_f32_split_kernel<<<(unsigned)((pieces + 255) / 256), 256, 0, s>>>(a, (uint4*)scratch, n_rows, k_dim, (int)k_pad,
                                                                          k_dim % 4 == 0 && aligned16(a));
    const int rc = st_launch_status();
    if (rc) return rc;
    const int grid = (int)(tiles < sms ? tiles : sms);
    if (nt <= 32) return gf_launch<32>(w_map, a_map, p, grid, status, s);
    if (nt <= 64) return gf_launch<64>(w_map, a_map, p, grid, status, s);
    return gf_launch<128>(w_map, a_map, p, grid, status, s);
}
