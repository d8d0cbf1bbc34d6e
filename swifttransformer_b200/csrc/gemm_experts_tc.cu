// The experts' products of a mixture on the 5th-generation tensor cores, bfloat16: for the rows offsets[g] .. offsets[g + 1] - 1
// of a list sorted by expert (see moe.cu)
//
//   c[row, n] = epilogue( sum_k a[arow, k] * w[g][n][k] )        arow = a_rows[row] / a_row_div, or the row itself
//
// with the epilogue of gemm_grouped.cu: act(product), or "gated": w[g] holds 2 * n_out rows, gate rows first, and
// c = act(gate) * up, both products rounded to bfloat16 first; with a limit the clamped unit of gated_clamped_act instead.
//
// One persistent block per SM walks through tiles of 128 rows x BN rows of w (gated: BN / 2 gate rows and the BN / 2 up rows
// beside them, so that one accumulator holds both).  Which tiles there are follows from the offsets on the device: expert by
// expert, and in an expert the row tiles of one column tile next to one another, so that the blocks that work at the same
// time share the weights' tile in the second-level cache and each weight comes from memory once.
//
// Warps: 0-3 read the accumulator (tcgen05.ld, a quarter of tensor memory each) and store; 4 copies weights, and rows of a
// where they are neighbours, by TMA boxes of 64 k (a in boxes of 32 rows, as many as the tile has); 5 issues tcgen05.mma;
// 6-9, where the rows are gathered, copy them by 16-byte asynchronous copies (tile::gather4 was measured at 20 cycles a row:
// 262 us for a product of 90 GFLOP that takes 109 this way).  Copies and products meet on a ring of stages; the accumulator
// is double-buffered in tensor memory, so that a tile is stored under the next one's products.  Rows of a tile past its
// expert's end hold other rows or what the shared memory held: a row of the product depends on its own row of a alone, and
// those are not stored.
//
// Bound by the tensor cores for prompts and by the weights' way from memory for few rows.  Measured on one B200 (with about
// 6 us of an empty launch between events, inputs not in cache; in brackets the mma.sync kernel with tiles of 64 x 64):
// 4000 items, 8 experts, 2048 -> 5504: 109 us = 880 TFLOP/s (481); 2752 -> 2048: 55 us = 920 TFLOP/s (252).  300 tokens x 2,
// 8 experts, gated 4096 -> 1024: 45 us (107).  38 items, 16 experts, 2048 -> 5504: 84 us, 361 MB = 4.6 TB/s (129).  16 items, 8
// experts, gated 2048 -> 512: 23 us (37).
//
// Waits are bounded: one that expires marks the block dead, `status` gets 5, and the block waits (again with a limit) for its
// copies under way, frees its tensor memory and leaves.
#include "tcgen05.cuh"
#include "tma_host.h"

#define GE_THREADS 192          // and 128 more where rows are gathered
#define GE_RING_BYTES (200 * 1024)
#define GE_STAGES(BN) (GE_RING_BYTES / (GE_BM * 128 + (BN) * 128) > GE_MAX_STAGES ? GE_MAX_STAGES : GE_RING_BYTES / (GE_BM * 128 + (BN) * 128))
#define GE_BM 128
#define GE_BK 64
#define GE_MAX_STAGES 8
#define GE_MAX_EXPERTS 1024

struct ExpertsShape {
    int n_experts, n_out, k_dim, gated, act, ldc, a_row_div, vec;
    float limit, alpha, shift;      // limit > 0: g = min(gate, limit), u = clamp(up, -limit, limit), c = g sigmoid(alpha g) (u + shift)
    const int* offsets;
    const int* a_rows;       // null: the rows of a are in sorted order
};

__device__ __forceinline__ void ge_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(mbar) : "memory");
}
// 8 consecutive float columns of this thread's lane of tensor memory, as tc_ld32
__device__ __forceinline__ void ge_ld8(uint32_t taddr, float* v) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr) : "memory");
}
// v / (1 + exp(-v)) of eight numbers side by side: the quotient by the fast division and one step of residual correction
// (chunks.cuh names the method), which gives the divided number's bits wherever the residual is a number.  As divisions they ran one after
// the other: 360 clocks each
__device__ __forceinline__ void ge_silu8(float* v) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float d = 1.f + expf(-v[j]), sc = d > 1e30f ? 5.421010862427522e-20f : 1.f;       // (2^-64: the fast one ends at 2^126)
        const float r = __fdividef(1.f, d * sc) * sc, q = v[j] * r, rest = fmaf(-q, d, v[j]);
        v[j] = rest < 0.f || rest > 0.f ? fmaf(rest, r, q) : q;
    }
}
// the clamped unit of eight gates v and ups u, the quotients as in ge_silu8
__device__ __forceinline__ void ge_clamped8(float* v, const float* u, float limit, float alpha, float shift) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float g = fminf(v[j], limit), up = fminf(fmaxf(u[j], -limit), limit);
        const float d = 1.f + expf(-alpha * g), sc = d > 1e30f ? 5.421010862427522e-20f : 1.f;
        const float r = __fdividef(1.f, d * sc) * sc, q = g * r, rest = fmaf(-q, d, g);
        v[j] = (rest < 0.f || rest > 0.f ? fmaf(rest, r, q) : q) * (up + shift);
    }
}
__device__ __forceinline__ void ge_act8(float* v, int act) {
    if (act == 4) ge_silu8(v);
    else if (act) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = apply_act(v[j], act);
    }
}

struct ExpertsTile {
    int expert, row0, rows, n0;
};

// tile number -> expert, rows and first column; `before` [n_experts + 1]: row tiles in front of each expert
__device__ __forceinline__ ExpertsTile ge_tile(int tile, int n_tiles_n, int bn_out, const int* before, const ExpertsShape& sh) {
    int lo = 0, hi = sh.n_experts;                       // the last expert whose tiles begin at or before this one
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (before[mid] * n_tiles_n <= tile) lo = mid; else hi = mid;
    }
    const int first = before[lo], mt = before[lo + 1] - first;
    const int local = tile - first * n_tiles_n;
    ExpertsTile t;
    t.expert = lo;
    t.n0 = (local / mt) * bn_out;
    const int begin = __ldcg(sh.offsets + lo), end = __ldcg(sh.offsets + lo + 1);
    t.row0 = begin + (local % mt) * GE_BM;
    t.rows = min(GE_BM, end - t.row0);
    return t;
}

template <int BN, bool GATHER>
__global__ void __launch_bounds__(GE_THREADS + (GATHER ? 128 : 0), 1)
gemm_experts_tc_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap a_map,
                       const bf16* __restrict__ a, bf16* __restrict__ c, const ExpertsShape sh, int* status) {
    extern __shared__ unsigned char ge_raw[];
    __shared__ __align__(8) unsigned long long s_full[GE_MAX_STAGES], s_empty[GE_MAX_STAGES], s_done[2], s_free[2];
    __shared__ uint32_t s_tmem;
    __shared__ int s_dead, s_issued;
    __shared__ int s_before[GE_MAX_EXPERTS + 1];
    constexpr uint32_t A_BYTES = GE_BM * 128, W_BYTES = BN * 128, STAGE = A_BYTES + W_BYTES;
    constexpr int TMEM_COLS = 2 * BN, stages = GE_STAGES(BN);
    const uint32_t base = (tc_smem(ge_raw) + 1023u) & ~1023u;
    const int tid = threadIdx.x, warp = tc_warp(), lane = tid & 31;
    volatile int* dead = &s_dead;
    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            tc_mbar_init(tc_smem(&s_full[s]), GATHER ? 129 : 1);
            tc_mbar_init(tc_smem(&s_empty[s]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            tc_mbar_init(tc_smem(&s_done[i]), 1);
            tc_mbar_init(tc_smem(&s_free[i]), 4);
        }
        tc_mbar_init_fence();
        s_dead = 0;
        s_issued = 0;
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     ::"r"(tc_smem(&s_tmem)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    __syncthreads();
    ST_PDL_WAIT();
    ST_PDL_TRIGGER();                                         // behind the allocation
    if (warp == 0) {
        int run = 0;
        for (int e0 = 0; e0 < sh.n_experts; e0 += 32) {
            const int e = e0 + lane;
            int mt = 0;
            if (e < sh.n_experts) mt = (__ldcg(sh.offsets + e + 1) - __ldcg(sh.offsets + e) + GE_BM - 1) / GE_BM;
            int sum = mt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += up;
            }
            if (e < sh.n_experts) s_before[e] = run + sum - mt;
            run += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) s_before[sh.n_experts] = run;
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = s_tmem;
    const int bn_out = sh.gated ? BN / 2 : BN;
    const int n_tiles_n = (sh.n_out + bn_out - 1) / bn_out;
    const int n_tiles = s_before[sh.n_experts] * n_tiles_n;
    const int n_k = (sh.k_dim + GE_BK - 1) / GE_BK;

    if (warp == 4) {
        // ---- weights, and rows of a that are neighbours
        const int w_rows = sh.gated ? 2 * sh.n_out : sh.n_out;
        int s = 0, turn = 0, it = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && tile < n_tiles; tile += gridDim.x) {
            const ExpertsTile t = ge_tile(tile, n_tiles_n, bn_out, s_before, sh);
            const int r0 = t.expert * w_rows + t.n0;
            const int boxes = GATHER ? 0 : (t.rows + 31) / 32;
            for (int k = 0; k < n_k; ++k) {
                if (turn > 0) ok = tc_wait_warp(tc_smem(&s_empty[s]), (turn - 1) & 1, dead);
                if (!ok) break;
                const uint32_t full = tc_smem(&s_full[s]), dst = base + s * STAGE + A_BYTES;
                if (tc_elect()) {
                    tc_mbar_expect_tx(full, W_BYTES + (uint32_t)boxes * 4096u);
                    tc_tma_load_2d(dst, &w_map, k * GE_BK, r0, full);
                    tc_tma_load_2d(dst + W_BYTES / 2, &w_map, k * GE_BK, sh.gated ? r0 + sh.n_out : r0 + BN / 2, full);
                    for (int b = 0; b < boxes; ++b)
                        tc_tma_load_2d(base + s * STAGE + b * 4096, &a_map, k * GE_BK, t.row0 + 32 * b, full);
                }
                ++it;
                if (++s == stages) { s = 0; ++turn; }
            }
        }
        if (lane == 0) s_issued = it;
    } else if (GATHER && warp >= 6) {
        // ---- gathered rows of a: a thread copies one 16-byte piece of every sixteenth row of the tile
        const int t128 = tid - GE_THREADS, piece = t128 & 7, r_first = t128 >> 3;
        const uint32_t at = (uint32_t)(r_first * 128 + ((piece ^ (r_first & 7)) << 4));      // rows 16 apart: the same swizzle
        int s = 0, turn = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && tile < n_tiles; tile += gridDim.x) {
            const ExpertsTile t = ge_tile(tile, n_tiles_n, bn_out, s_before, sh);
            const bf16* src[GE_BM / 16];
#pragma unroll
            for (int i = 0; i < GE_BM / 16; ++i) {
                const int row = t.row0 + min(r_first + 16 * i, t.rows - 1);
                src[i] = a + (size_t)(__ldcg(sh.a_rows + row) / sh.a_row_div) * sh.k_dim + piece * 8;
            }
            for (int k = 0; k < n_k; ++k) {
                if (turn > 0) ok = tc_wait_warp(tc_smem(&s_empty[s]), (turn - 1) & 1, dead);
                if (!ok) break;
                const bool in_k = k * GE_BK + piece * 8 < sh.k_dim;
                const uint32_t dst = base + s * STAGE + at;
#pragma unroll
                for (int i = 0; i < GE_BM / 16; ++i)
                    if (r_first + 16 * i < t.rows) tc_cp16(dst + i * 2048, in_k ? src[i] + k * GE_BK : a, in_k);
                // the thread's arrival when its copies have landed; the products' thread makes them visible to the tensor cores
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(tc_smem(&s_full[s])) : "memory");
                if (++s == stages) { s = 0; ++turn; }
            }
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
    } else if (warp == 5) {
        // ---- products
        const uint32_t idesc = tc_idesc(GE_BM, BN, 0, 0);
        int s = 0, turn = 0, i = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && tile < n_tiles; tile += gridDim.x, ++i) {
            const int buf = i & 1;
            if (i >= 2) ok = tc_wait_warp(tc_smem(&s_free[buf]), ((i >> 1) - 1) & 1, dead);
            if (!ok) break;
            tc_fence_after_sync();
            for (int k = 0; k < n_k; ++k) {
                ok = tc_wait_warp(tc_smem(&s_full[s]), turn & 1, dead);
                if (!ok) break;
                if (GATHER) tc_fence_async_smem();
                tc_fence_after_sync();
                const uint64_t da = tc_desc(base + s * STAGE, 16, 1024), dw = tc_desc(base + s * STAGE + A_BYTES, 16, 1024);
                if (tc_elect()) {
#pragma unroll
                    for (int kk = 0; kk < GE_BK / 16; ++kk)
                        tc_mma(tmem + buf * BN, da + ((kk * 32) >> 4), dw + ((kk * 32) >> 4), idesc, k > 0 || kk > 0);
                    tc_commit(tc_smem(&s_empty[s]));
                }
                __syncwarp();
                if (++s == stages) { s = 0; ++turn; }
            }
            if (tc_elect()) tc_commit(tc_smem(&s_done[buf]));
        }
    } else if (warp < 4) {
        // ---- epilogue: warp q holds rows 32 q .. 32 q + 31 of the tile, a thread its row
        int i = 0;
        for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++i) {
            const ExpertsTile t = ge_tile(tile, n_tiles_n, bn_out, s_before, sh);
            const int buf = i & 1;
            if (!tc_wait_warp(tc_smem(&s_done[buf]), (i >> 1) & 1, dead)) break;
            tc_fence_after_sync();
            const int r = warp * 32 + lane;
            const uint32_t t_row = tmem + buf * BN + ((uint32_t)(warp * 32) << 16);
            if (warp * 32 < t.rows) {
                bf16* dst = c + (size_t)(t.row0 + r) * sh.ldc + t.n0;
                const bool live = r < t.rows;
                // eight columns at a time and not unrolled: the activations' code is long, and a launch of few rows runs it
                // once (unrolled over 32 columns it took 11 us of a decode step's 30)
#pragma unroll 1
                for (int c0 = 0; c0 < bn_out; c0 += 8) {
                    if (t.n0 + c0 >= sh.n_out) break;
                    float v[8], u[8];
                    ge_ld8(t_row + c0, v);
                    if (sh.gated) ge_ld8(t_row + BN / 2 + c0, u);
                    tc_ld_wait();
                    if (sh.gated) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) v[j] = to_f32(from_f32<bf16>(v[j]));
                    }
                    // rows past the expert's end hold anything: a division of numbers out of its quick range takes the whole
                    // warp through the slow one, hundreds of clocks per column
                    if (!live) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) v[j] = 0.f;
                    }
                    if (sh.gated) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) u[j] = to_f32(from_f32<bf16>(u[j]));
                    }
                    if (sh.limit > 0.f) ge_clamped8(v, u, sh.limit, sh.alpha, sh.shift);
                    else {
                        ge_act8(v, sh.act);
                        if (sh.gated) {
#pragma unroll
                            for (int j = 0; j < 8; ++j) v[j] *= u[j];
                        }
                    }
                    if (live && sh.vec && t.n0 + c0 + 8 <= sh.n_out) {
                        uint4 p;
                        uint32_t* w4 = reinterpret_cast<uint32_t*>(&p);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
                            w4[e] = *reinterpret_cast<const uint32_t*>(&b);
                        }
                        *reinterpret_cast<uint4*>(dst + c0) = p;
                    } else if (live) {
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (t.n0 + c0 + j < sh.n_out) dst[c0 + j] = from_f32<bf16>(v[j]);
                    }
                    __syncwarp();                         // the next tcgen05.ld is the whole warp's
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) ge_arrive(tc_smem(&s_free[buf]));
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (s_dead && tid == 0) {
        // copies and products under way end before the block's memory is given up: a stage's boxes by its barrier (which
        // also wants the gathered rows; those have been waited for), the rest by time, a few milliseconds
        atomicExch(status, 5);
        if (!GATHER)
            for (int s = 0; s < stages && s < s_issued; ++s) tc_wait(tc_smem(&s_full[s]), ((s_issued - 1 - s) / stages) & 1);
        for (int i = 0; i < 20000; ++i) __nanosleep(100);
    }
    __syncthreads();
    if (warp == 5) {
        tc_fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// The rows of w in a tile (gated tiles count their gate and up rows).  The wider, the less a is read again; a launch has at
// least a row tile per expert that any item may go to.  Lines by measurement (us with 64 / 128 / 256 rows): the widest while
// every SM gets a tile (4000 items, 5504 rows: 254 / 152 / 102), then 128 while half of the SMs do (600 items on 8 experts, 2048
// gate and up rows: 59 / 45 / 53; 256 items on 16 experts, 1024: 25 / 21 / 25; 16 items on 8, 2048: 16 / 14 / 18; but 16 on 16, 1024
// of k = 512: 14.3 / 16.4 / 20.5), else 64 (16 items on 8, 1024: 23 / 25 / 29).  Over 650 products of 8 to 128 experts the choice is 2 %
// behind the best width on average; counting only the experts that items are likely to hit, or the rounds of tiles, gained nothing.
static int ge_pick_bn(int n_items, int n_experts, int w_rows, int sms) {
    int row_tiles = (n_items + GE_BM - 1) / GE_BM;
    if (row_tiles < n_experts) row_tiles = n_items < n_experts ? n_items : n_experts;
    auto tiles = [&](int bn) { return (long long)row_tiles * ((w_rows + bn - 1) / bn); };
    return tiles(256) >= sms ? 256 : 2 * tiles(128) >= sms ? 128 : 64;
}

template <int BN, bool GATHER>
static int ge_launch(const CUtensorMap& w_map, const CUtensorMap& a_map, const bf16* a, bf16* c, ExpertsShape sh,
                     long long max_tiles, int* status, cudaStream_t s) {
    constexpr size_t smem = (size_t)GE_STAGES(BN) * (GE_BM * 128 + BN * 128) + 1024;
    auto kernel = gemm_experts_tc_kernel<BN, GATHER>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const long long grid = max_tiles < st_sm_count() ? max_tiles : st_sm_count();
    return st_launch_pdl("gemm_experts_tc", kernel, dim3((unsigned)grid), dim3(GE_THREADS + (GATHER ? 128 : 0)), smem, s, w_map,
                         a_map, a, c, sh, status);
}

ST_EXPORT int st_gemm_experts_tc_applies(int n_experts, int k_dim) {
    return n_experts > 0 && n_experts <= GE_MAX_EXPERTS && k_dim > 0 && k_dim % 8 == 0;
}

// a [a_n_rows, k_dim], w [n_experts, w_rows, k_dim] (w_rows = n_out, twice that with `gated`), c [n_items, n_out], all bfloat16
// and contiguous; offsets [n_experts + 1]; a_rows [n_items] or null (a's rows are then the items in sorted order).
// tile_bn: rows of w per tile (64, 128, 256), 0: chosen here.  limit > 0 (gated): the clamped unit with alpha and shift, act is not read.
ST_EXPORT int st_gemm_experts_tc(const void* a, long long a_n_rows, const void* w, void* c, int n_experts, int n_items, int n_out,
                                 int k_dim, int gated, int act, const int* offsets, const int* a_rows, int a_row_div, int tile_bn,
                                 int* status, void* stream, float limit, float alpha, float shift) {
    if (n_items <= 0 || n_out <= 0) return 0;
    if (!offsets || !status || (a_rows && a_row_div <= 0) || a_n_rows <= 0) return ST_ERR_BAD_ARG;
    if (limit > 0.f && !gated) return ST_ERR_BAD_ARG;
    if (!st_gemm_experts_tc_applies(n_experts, k_dim) || !aligned16(a) || !aligned16(w)) return ST_ERR_BAD_SIZE;
    const int w_rows = gated ? 2 * n_out : n_out;
    if ((long long)n_experts * w_rows > 0x7fffffffLL || a_n_rows > 0x7fffffffLL) return ST_ERR_TOO_LARGE;
    const int bn = tile_bn ? tile_bn : ge_pick_bn(n_items, n_experts, w_rows, st_sm_count());
    if (bn != 64 && bn != 128 && bn != 256) return ST_ERR_BAD_ARG;
    const unsigned long long wd[2] = {(unsigned long long)k_dim, (unsigned long long)n_experts * w_rows};
    const unsigned long long ad[2] = {(unsigned long long)k_dim, (unsigned long long)a_n_rows};
    const unsigned wb[2] = {GE_BK, (unsigned)bn / 2}, ab[2] = {GE_BK, 32};
    CUtensorMap w_map, a_map;
    if (st_tma_encode_bf16(&w_map, w, 2, wd, wb) || st_tma_encode_bf16(&a_map, a, 2, ad, ab)) return ST_ERR_BAD_ARG;
    ExpertsShape sh;
    sh.n_experts = n_experts; sh.n_out = n_out; sh.k_dim = k_dim; sh.gated = gated; sh.act = act; sh.ldc = n_out;
    sh.limit = limit; sh.alpha = alpha; sh.shift = shift;
    sh.a_row_div = a_row_div; sh.vec = n_out % 8 == 0 && aligned16(c); sh.offsets = offsets; sh.a_rows = a_rows;
    const int bn_out = gated ? bn / 2 : bn;
    const long long max_tiles = ((n_items + GE_BM - 1) / GE_BM + (long long)n_experts) * ((n_out + bn_out - 1) / bn_out);
    if (max_tiles > 0x3fffffffLL) return ST_ERR_TOO_LARGE;
    cudaStream_t s = (cudaStream_t)stream;
#define GE_LAUNCH(BN)                                                                                                  \
    return a_rows ? ge_launch<BN, true>(w_map, a_map, (const bf16*)a, (bf16*)c, sh, max_tiles, status, s)              \
                  : ge_launch<BN, false>(w_map, a_map, (const bf16*)a, (bf16*)c, sh, max_tiles, status, s)
    if (bn == 64) GE_LAUNCH(64);
    if (bn == 128) GE_LAUNCH(128);
    GE_LAUNCH(256);
#undef GE_LAUNCH
}
