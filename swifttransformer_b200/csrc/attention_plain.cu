// Plain paged attention: one thread block per (query token, head), for any
// head size, page size, number of heads and groups, in float or bfloat16
// storage with float arithmetic throughout.
//
// The query at position p of a request attends the keys lo..p of that
// request, lo = max(0, p - window + 1) (window <= 0: all keys), read from the
// pages its block table names; the step's own keys have been written before.
// Keys are visited in tiles of KT aligned to absolute positions and reduced in
// a fixed order, so the result for a position does not depend on how the
// request was cut into steps or on what else is in the batch.
//
// Float storage with rows of whole 16-byte pieces goes to attention_f32_kernel and attention_f32_few_kernel (below), which give
// the same bits; every other size and bfloat16 storage to attention_plain_kernel.
//
// Formulas: src/csrc/kernel/fused_decoding_stage_attention_mha.cu:159-252
// (scores, softmax) and :254-318 (weighted sum of values); the prompt kernel
// src/csrc/kernel/fused_context_stage_attention.cu:226-404 computes the same
// per row.  Not taken over: the -10000 additive mask and the +1e-6 in the
// denominator; masked keys are simply not visited.
#include "common.cuh"

#define KT 128  // keys per tile == threads per block

template <typename T>
__global__ void __launch_bounds__(KT)
attention_plain_kernel(const T* __restrict__ q, const T* __restrict__ pool, T* __restrict__ out,
                       const int* __restrict__ positions, const int* __restrict__ seq_of_token,
                       const int* __restrict__ slots, const int* __restrict__ block_table, int max_pages,
                       int n_layers, int layer, int nh, int nkv, int d, int page_size, float scale, int window,
                       int* __restrict__ status) {
    extern __shared__ float smem[];
    float* sq = smem;        // [d] query, pre-scaled
    float* sp = smem + d;    // [KT] probabilities of the tile
    __shared__ float scratch[32];
    const int t = blockIdx.x, h = blockIdx.y;
    const int kvh = h / (nh / nkv);
    const int pos = positions[t];
    if (pos < 0) return;   // padding token of a fixed-shape step
    const int slot = slots[seq_of_token[t]];
    const int* bt = block_table + (size_t)slot * max_pages;
    for (int e = threadIdx.x; e < d; e += blockDim.x) sq[e] = to_f32(q[((size_t)t * nh + h) * d + e]) * scale;
    __syncthreads();
    const int lo = window > 0 ? max(0, pos - window + 1) : 0;
    const int hi = pos + 1;
    const int ndim = (d + KT - 1) / KT;   // output dims per thread (d <= 2*KT is enforced by the launcher)
    float acc[2] = {0.f, 0.f};
    float m = -INFINITY, l = 0.f;
    for (int base = (lo / KT) * KT; base < hi; base += KT) {
        const int j = base + threadIdx.x;
        float s = -INFINITY;
        if (j >= lo && j < hi) {
            const int page = bt[j / page_size];
            if (page >= 0) {     // a hole in the block table: the key is dropped, no access before the pool
                const T* krow = pool + (((((size_t)page * n_layers + layer) * 2 + 0) * nkv + kvh) * page_size + j % page_size) * d;
                float dot = 0.f;
                for (int e = 0; e < d; ++e) dot += sq[e] * to_f32(krow[e]);
                s = dot;
            } else if (status) {
                *status = 1;     // reported to the host: the step's bookkeeping is broken
            }
        }
        const float tile_max = block_max(s, scratch);
        const float m_new = fmaxf(m, tile_max);
        const float p = (j >= lo && j < hi) ? expf(s - m_new) : 0.f;
        const float tile_sum = block_sum(p, scratch);
        const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
        l = l * corr + tile_sum;
        m = m_new;
        sp[threadIdx.x] = p;
        __syncthreads();
        const int j_end = min(KT, hi - base);
        const int j_begin = max(0, lo - base);
        for (int c = 0; c < ndim; ++c) {
            const int e = threadIdx.x + c * KT;
            if (e < d) {
                float a = acc[c] * corr;
                for (int jj = j_begin; jj < j_end; ++jj) {
                    const int key = base + jj;
                    const int page = bt[key / page_size];
                    if (page < 0) continue;      // dropped above: its weight is zero
                    const T* vrow = pool + (((((size_t)page * n_layers + layer) * 2 + 1) * nkv + kvh) * page_size + key % page_size) * d;
                    a += sp[jj] * to_f32(vrow[e]);
                }
                acc[c] = a;
            }
        }
        __syncthreads();
    }
    const float inv = l > 0.f ? 1.0f / l : 0.f;      // no key at all (every page missing): zeros, not NaN
    for (int c = 0; c < ndim; ++c) {
        const int e = threadIdx.x + c * KT;
        if (e < d) out[((size_t)t * nh + h) * d + e] = from_f32<T>(acc[c] * inv);
    }
}

// ---- float storage, tiles of query rows -----------------------------------------------------------------------
// A block serves one head of the tokens 32 i .. 32 i + 31 of the step, one run of neighbouring positions of one request
// after the other (with gridDim.z > 1 every gridDim.z-th run: steps of single tokens have a run per token).  Every sum has
// the order of attention_plain_kernel: scores and weighted values are chains over ascending dimensions / keys, a tile's
// exponentials are added over 32 lanes, then over the four groups of 32 keys; so neither the way of a run through
// this kernel nor the length of the run changes a row's bits.
//
// A run of several tokens: scores of its 32 rows x 32 keys (4 x 2 per thread), four times per tile of 128 keys; then the rows'
// softmax by a warp per eight rows; then rows x values (4 rows x 4 dimensions per thread and 64 dimensions).  Key
// and value rows come 32 at a time through three stages of shared memory filled by 16-byte asynchronous copies.  Bound by
// shared memory (six reads of two cycles per 32 multiply-adds of a warp for the scores).
// A run of one token: a thread per key reads its row from memory; the tile's values arrive meanwhile in shared memory.
// (The instances for 64 and 128 dimensions spill 76 and 56 bytes a thread at the registers of four and three blocks per SM.)
// Three prompts of 700 tokens in all, 32 heads of 64: 89 us (112 with the tiles in ascending order, once per head); the general
// kernel 1089 (each of its blocks reads all its keys again, the lanes of a warp in 32 different rows at once).
#define AF_ROWS 32
#define AF_SUB 32
#define AF_STAGES 3
#define AF_LDS (KT + 4)

__device__ __forceinline__ void af_cp16(float* dst, const float* src, bool ok) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(ok ? 16 : 0));
}
__device__ __forceinline__ void af_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void af_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

struct AttentionF32 {
    const float* q;
    const float* pool;
    float* out;
    const int *positions, *seq_of_token, *slots, *block_table;
    int n_tokens, max_pages, n_layers, layer, nh, nkv, d, page_size, window;
    float scale;
    int* status;
    int n_seqs;
};

// the pool's row of key `key` of a request, -1: none (past the run's range, or a hole in the block table: reported)
__device__ __forceinline__ long long af_row(const AttentionF32& p, const int* bt, int kvh, int key, int lo, int hi) {
    if (key < lo || key >= hi) return -1;
    const int page = bt[key / p.page_size];
    if (page < 0) {
        if (p.status) *p.status = 1;
        return -1;
    }
    return ((((long long)page * p.n_layers + p.layer) * 2) * p.nkv + kvh) * p.page_size + key % p.page_size;
}

// one token: threads are keys for the scores, dimensions for the values.  A tile's values pass through GROUPS places of AF_SUB
// rows: all of them at once (4), or two by two (2), which leaves room for more blocks on an SM
template <int GROUPS>
__device__ __forceinline__ void af_single(const AttentionF32& p, float* smem, long long* rows, float* scratch, int t, int h,
                                          int kvh, int pos, const int* bt) {
    static_assert(KT / AF_SUB == 4 && (GROUPS == 2 || GROUPS == 4), "a tile is four groups of keys");
    const int d = p.d, tid = threadIdx.x;
    float* sv = smem;                    // [GROUPS][AF_SUB][d] values of the tile
    float* sq = smem + GROUPS * AF_SUB * d;     // [d] scaled query
    float* sp = sq + d;                  // [KT] weights
    const float* q = p.q + ((size_t)t * p.nh + h) * d;
    const int lo = p.window > 0 ? max(0, pos - p.window + 1) : 0, hi = pos + 1;
    const size_t v_off = (size_t)p.nkv * p.page_size * d;
    for (int e = tid; e < d; e += KT) sq[e] = q[e] * p.scale;
    const int pieces = d / 4;
    float acc[2] = {0.f, 0.f};
    float m = -INFINITY, l = 0.f;
    for (int base = (lo / KT) * KT; base < hi; base += KT) {
        const long long row = af_row(p, bt, kvh, base + tid, lo, hi);
        rows[tid] = row;
        __syncthreads();                 // the rows' places; also: the tile before is done with the values' memory
        const int j_begin = max(0, lo - base), j_end = min(KT, hi - base);
        auto copy = [&](float* dst, int a, int b) {      // the values of keys a .. b - 1
            for (int i = tid + a * pieces; i < b * pieces; i += KT) {
                const long long r = rows[i / pieces];
                af_cp16(dst + i * 4, r >= 0 ? p.pool + r * d + v_off + (i % pieces) * 4 : p.pool, r >= 0);
            }
            af_commit();
        };
        auto group = [&](int g) { return sv + (g % GROUPS - g) * AF_SUB * d; };      // where key 0 would be
        auto copy_group = [&](int g) { copy(group(g), max(j_begin, g * AF_SUB), min(j_end, (g + 1) * AF_SUB)); };
        if constexpr (GROUPS == 4) {
            copy(sv, j_begin, j_end);
        } else {
            copy_group(0);
            copy_group(1);
        }
        float s = -INFINITY;
        if (row >= 0) {
            const float4* k = reinterpret_cast<const float4*>(p.pool + row * d);
            float dot = 0.f;
#pragma unroll 8
            for (int e = 0; e < pieces; ++e) {
                const float4 kv = k[e], qv = *reinterpret_cast<const float4*>(sq + 4 * e);
                dot = fmaf(qv.x, kv.x, dot); dot = fmaf(qv.y, kv.y, dot); dot = fmaf(qv.z, kv.z, dot); dot = fmaf(qv.w, kv.w, dot);
            }
            s = dot;
        }
        const float m_new = fmaxf(m, block_max(s, scratch));
        const float w = row >= 0 ? expf(s - m_new) : 0.f;
        const float tile_sum = block_sum(w, scratch);
        const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
        l = fmaf(l, corr, tile_sum);
        m = m_new;
        sp[tid] = w;
        auto add = [&](const float* v, int a, int b, float corr) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int e = tid + c * KT;
                if (e < d) {
                    float x = acc[c] * corr;
                    int j = a;
                    for (; j < b && (j & 3); ++j) x = fmaf(sp[j], v[j * d + e], x);
#pragma unroll 4
                    for (; j + 4 <= b; j += 4) {
                        const float4 w4 = *reinterpret_cast<const float4*>(sp + j);
                        x = fmaf(w4.x, v[j * d + e], x);
                        x = fmaf(w4.y, v[(j + 1) * d + e], x);
                        x = fmaf(w4.z, v[(j + 2) * d + e], x);
                        x = fmaf(w4.w, v[(j + 3) * d + e], x);
                    }
                    for (; j < b; ++j) x = fmaf(sp[j], v[j * d + e], x);
                    acc[c] = x;
                }
            }
        };
        if constexpr (GROUPS == 4) {
            af_wait<0>();
            __syncthreads();
            add(sv, j_begin, j_end, corr);
        } else {
            for (int g = 0; g < 4; ++g) {
                af_wait<1>();            // of two groups under way the first has landed
                __syncthreads();
                add(group(g), max(j_begin, g * AF_SUB), min(j_end, (g + 1) * AF_SUB), g == 0 ? corr : 1.f);
                if (g < 2 && (g + 2) * AF_SUB < j_end) {
                    __syncthreads();     // everyone is done with the group whose place is filled next
                    copy_group(g + 2);
                } else {
                    af_commit();
                }
            }
        }
    }
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    for (int c = 0; c < 2; ++c) {
        const int e = tid + c * KT;
        if (e < d) p.out[((size_t)t * p.nh + h) * d + e] = acc[c] * inv;
    }
    __syncthreads();                     // shared memory is free for the next run
}

// Steps of few tokens (af_few): a block per (token, head), whatever runs there are.  At most 2 x 32 value rows in shared memory, so that
// many blocks share an SM; a tile of 32 query rows, or a tile's values at once, leave room for two at 128 dimensions.
__global__ void __launch_bounds__(KT, 8)
attention_f32_few_kernel(const AttentionF32 p) {
    extern __shared__ __align__(16) float smem[];
    __shared__ long long rows[KT];
    __shared__ float scratch[32];
    const int h = blockIdx.x % p.nh, t = p.n_tokens - 1 - blockIdx.x / p.nh;
    const int pos = p.positions[t];
    if (pos < 0) return;
    af_single<2>(p, smem, rows, scratch, t, h, h / (p.nh / p.nkv), pos, p.block_table + (size_t)p.slots[p.seq_of_token[t]] * p.max_pages);
}

// n tokens t0 .. t0 + n - 1 at positions pos0 .. pos0 + n - 1; NI: 64-wide blocks of dimensions
template <int NI>
__device__ __forceinline__ void af_tile(const AttentionF32& p, float* smem, long long* rows, float* s_corr, int t0, int n, int h,
                                        int kvh, int pos0, const int* bt) {
    const int d = p.d, ld = d + 4, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* ring = smem;                                  // [AF_STAGES][AF_SUB][ld]
    float* sq = ring + AF_STAGES * AF_SUB * ld;          // [AF_ROWS][ld] scaled queries
    float* S = sq + AF_ROWS * ld;                        // [AF_ROWS][AF_LDS] scores, then weights
    const int pieces = d / 4;
    const int kmin = p.window > 0 ? max(0, pos0 - p.window + 1) : 0, kmax = pos0 + n;
    const int lo_last = p.window > 0 ? max(0, pos0 + n - p.window) : 0;
    const size_t v_off = (size_t)p.nkv * p.page_size * d;
    for (int i = tid; i < AF_ROWS * pieces; i += KT) {
        const int r = i / pieces, e = (i % pieces) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < n) v = *reinterpret_cast<const float4*>(p.q + ((size_t)(t0 + r) * p.nh + h) * d + e);
        *reinterpret_cast<float4*>(sq + r * ld + e) = make_float4(v.x * p.scale, v.y * p.scale, v.z * p.scale, v.w * p.scale);
    }
    const int base0 = (kmin / KT) * KT, n_tiles = (kmax - base0 + KT - 1) / KT;
    // the copies in order: per tile its live groups of 32 keys, then the same groups' values
    int c_tile = 0, c_sub = 0, c_v = 0, c_stage = 0;
    auto sub_live = [&](int tile, int sub) {
        const int b = base0 + tile * KT + sub * AF_SUB;
        return b < kmax && b + AF_SUB > kmin;
    };
    auto look_up = [&](int tile) { rows[(tile & 1) * KT + tid] = af_row(p, bt, kvh, base0 + tile * KT + tid, kmin, kmax); };
    auto advance = [&]() {               // to the next live group
        do {
            if (++c_sub == KT / AF_SUB) {
                c_sub = 0;
                if (c_v) ++c_tile;
                c_v ^= 1;
            }
        } while (c_tile < n_tiles && !sub_live(c_tile, c_sub));
    };
    auto copy_next = [&]() {
        if (c_tile < n_tiles) {
            float* dst = ring + c_stage * AF_SUB * ld;
            const long long* rw = rows + (c_tile & 1) * KT + c_sub * AF_SUB;
            const float* src = p.pool + (c_v ? v_off : 0);
            for (int i = tid; i < AF_SUB * pieces; i += KT) {
                const int r = i / pieces, e = (i % pieces) * 4;
                const long long row = rw[r];
                af_cp16(dst + r * ld + e, row >= 0 ? src + row * d + e : p.pool, row >= 0);
            }
            advance();
            if (++c_stage == AF_STAGES) c_stage = 0;
        }
        af_commit();
    };
    look_up(0);
    if (!sub_live(0, 0)) advance();
    __syncthreads();
    copy_next();
    copy_next();
    // a thread's four rows rg + 8 i, its two keys kl + 16 j of a group, its dimensions 4 kl + 64 b ..; lanes l and l ^ 1 share
    // the keys' (values') 16 bytes, lanes l and l ^ 2 the queries' (weights'): two cycles of shared memory per read
    const int rg = warp * 2 + (lane & 1), kl = lane >> 1;
    float acc[NI][4][4];
#pragma unroll
    for (int b = 0; b < NI; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[b][i][e] = 0.f;
    float m[8], l[8];                    // of rows 8 warp + i, the same in every lane
#pragma unroll
    for (int i = 0; i < 8; ++i) { m[i] = -INFINITY; l[i] = 0.f; }
    int stage = 0;
    for (int tile = 0; tile < n_tiles; ++tile) {
        const int base = base0 + tile * KT;
        bool looked = false;
        for (int sub = 0; sub < KT / AF_SUB; ++sub) {
            if (!sub_live(tile, sub)) continue;
            af_wait<1>();
            __syncthreads();             // the group has landed; everyone is done with the stage that is filled next
            // the places of the next tile's rows: written when all copies of the tile before last have been issued
            if (!looked && tile + 1 < n_tiles) { look_up(tile + 1); looked = true; __syncthreads(); }
            copy_next();
            const float* K = ring + stage * AF_SUB * ld;
            float s[4][2] = {};
#pragma unroll 4
            for (int e = 0; e < pieces; ++e) {
                float4 qv[4], kv[2];
#pragma unroll
                for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const float4*>(sq + (rg + 8 * i) * ld + 4 * e);
#pragma unroll
                for (int j = 0; j < 2; ++j) kv[j] = *reinterpret_cast<const float4*>(K + (kl + 16 * j) * ld + 4 * e);
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        s[i][j] = fmaf(qv[i].x, kv[j].x, s[i][j]);
                        s[i][j] = fmaf(qv[i].y, kv[j].y, s[i][j]);
                        s[i][j] = fmaf(qv[i].z, kv[j].z, s[i][j]);
                        s[i][j] = fmaf(qv[i].w, kv[j].w, s[i][j]);
                    }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) S[(rg + 8 * i) * AF_LDS + sub * AF_SUB + kl + 16 * j] = s[i][j];
            if (++stage == AF_STAGES) stage = 0;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = warp * 8 + i, pos = pos0 + r;
            const int lo = p.window > 0 ? max(0, pos - p.window + 1) : 0;
            float x[4];
            bool ok[4];
            float mx = -INFINITY;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const int key = base + g * 32 + lane;
                ok[g] = r < n && key >= lo && key <= pos && rows[(tile & 1) * KT + g * 32 + lane] >= 0;
                x[g] = ok[g] ? S[r * AF_LDS + g * 32 + lane] : -INFINITY;
                mx = fmaxf(mx, x[g]);
            }
            const float m_new = fmaxf(m[i], warp_max(mx));
            float tile_sum = 0.f;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const float w = ok[g] ? expf(x[g] - m_new) : 0.f;
                S[r * AF_LDS + g * 32 + lane] = w;
                tile_sum += warp_sum(w);
            }
            const float corr = (m[i] == -INFINITY) ? 0.f : expf(m[i] - m_new);
            l[i] = fmaf(l[i], corr, tile_sum);
            m[i] = m_new;
            if (lane == 0) s_corr[r] = corr;
        }
        bool first = true;
        for (int sub = 0; sub < KT / AF_SUB; ++sub) {
            if (!sub_live(tile, sub)) continue;
            af_wait<1>();
            __syncthreads();
            copy_next();
            if (first) {
                first = false;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float corr = s_corr[rg + 8 * i];
#pragma unroll
                    for (int b = 0; b < NI; ++b)
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[b][i][e] *= corr;
                }
            }
            const float* V = ring + stage * AF_SUB * ld;
            const int kb = base + sub * AF_SUB;
            // a group that every row sees whole; in the others a key is added to the rows that see it (a row's sum must
            // not meet the values of keys it does not see, whatever they are)
            const bool whole = kb + AF_SUB - 1 <= pos0 && kb >= lo_last;
            for (int j = 0; j < AF_SUB; j += 4) {
                float4 w[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(S + (rg + 8 * i) * AF_LDS + sub * AF_SUB + j);
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    const int key = kb + j + jj;
                    bool sees[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int pos = pos0 + rg + 8 * i;
                        sees[i] = whole || (key <= pos && (p.window <= 0 || key > pos - p.window));
                    }
#pragma unroll
                    for (int b = 0; b < NI; ++b) {
                        if (4 * kl + 64 * b >= d) continue;
                        const float4 v = *reinterpret_cast<const float4*>(V + (j + jj) * ld + 4 * kl + 64 * b);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float wi = jj == 0 ? w[i].x : jj == 1 ? w[i].y : jj == 2 ? w[i].z : w[i].w;
                            if (sees[i]) {
                                acc[b][i][0] = fmaf(wi, v.x, acc[b][i][0]);
                                acc[b][i][1] = fmaf(wi, v.y, acc[b][i][1]);
                                acc[b][i][2] = fmaf(wi, v.z, acc[b][i][2]);
                                acc[b][i][3] = fmaf(wi, v.w, acc[b][i][3]);
                            }
                        }
                    }
                }
            }
            if (++stage == AF_STAGES) stage = 0;
        }
    }
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int i = 0; i < 8; ++i) s_corr[warp * 8 + i] = l[i] > 0.f ? 1.0f / l[i] : 0.f;
    af_wait<0>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = rg + 8 * i;
        if (r >= n) continue;
        const float inv = s_corr[r];
#pragma unroll
        for (int b = 0; b < NI; ++b)
            if (4 * kl + 64 * b < d)
                *reinterpret_cast<float4*>(p.out + ((size_t)(t0 + r) * p.nh + h) * d + 4 * kl + 64 * b) =
                    make_float4(acc[b][i][0] * inv, acc[b][i][1] * inv, acc[b][i][2] * inv, acc[b][i][3] * inv);
    }
    __syncthreads();
}

template <int NI>
__global__ void __launch_bounds__(KT, NI == 1 ? 4 : NI == 2 ? 3 : 1)
attention_f32_kernel(const AttentionF32 p) {
    extern __shared__ __align__(16) float smem[];
    __shared__ long long rows[2 * KT];
    __shared__ float scratch[32];
    // all heads of a tile of tokens before the next tile, a request's last tokens, who see the most keys, first
    const int lane = threadIdx.x & 31, h = blockIdx.x % p.nh, kvh = h / (p.nh / p.nkv);
    const int first = (gridDim.x / p.nh - 1 - blockIdx.x / p.nh) * AF_ROWS, t = first + lane;
    const int pos = t < p.n_tokens ? p.positions[t] : -1;
    const int seq = pos >= 0 ? p.seq_of_token[t] : -1;
    // runs: neighbouring tokens of one request at neighbouring positions (each warp finds the same ones)
    const int pos_before = __shfl_up_sync(0xffffffffu, pos, 1), seq_before = __shfl_up_sync(0xffffffffu, seq, 1);
    const unsigned alive = __ballot_sync(0xffffffffu, pos >= 0);
    unsigned starts = __ballot_sync(0xffffffffu, pos >= 0 && (lane == 0 || seq != seq_before || pos != pos_before + 1));
    for (int k = 0; starts; ++k) {
        const int at = __ffs(starts) - 1;
        starts &= starts - 1;
        const unsigned ends = (~alive | starts) & ~((2u << at) - 1u);        // what stops the run: the next start, a gap, the end
        const int stop = ends ? __ffs(ends) - 1 : 32;
        if (k % gridDim.z != blockIdx.z) continue;
        const int pos0 = __shfl_sync(0xffffffffu, pos, at), s0 = __shfl_sync(0xffffffffu, seq, at);
        const int* bt = p.block_table + (size_t)p.slots[s0] * p.max_pages;
        if (stop - at == 1) af_single<KT / AF_SUB>(p, smem, rows, scratch, first + at, h, kvh, pos0, bt);
        else af_tile<NI>(p, smem, rows, scratch, first + at, stop - at, h, kvh, pos0, bt);
    }
}

// Whether every token of the step is a block's of its own: (token, head) pairs per multiprocessor times tokens per request up to
// 30000 / dimensions.  A tile reads its keys once for all its rows but takes as long for two tokens as for 32, and its shared
// memory leaves room for four, two or one block per SM (64, 128, 256 dimensions).  us on one B200, tiles / tokens (general kernel),
// 32 heads: 64 dimensions, one request of 16 tokens at 0 / 100 / 1000 earlier ones 20 / 10 (20), 33 / 16 (88), 199 / 84 (653);
// 4 requests of 16 20 / 16 (27), 47 / 35, 293 / 230; 4 of 32 25 / 27 (57), 47 / 61, 285 / 385; 128 dimensions, 16 of 4 37 / 22
// (20), 88 / 64, 698 / 473; 16 of 8 45 / 35 (35), 121 / 108, 813 / 883; one of 64 behind 1000 291 / 447; 256 dimensions, 16 heads,
// 16 of 4 45 / 31 (27), 4 of 32 41 / 55 (102).  Steps of single tokens stay with the tiles' kernel, whose values arrive at once.
static bool af_few(const AttentionF32& p) {
    if (p.n_seqs <= 0 || p.n_tokens <= p.n_seqs) return false;
    const int limit = 30000 / (p.d > 64 ? p.d : 64);
    return (double)p.n_tokens * p.nh * p.n_tokens <= (double)limit * st_sm_count() * p.n_seqs;
}

static int attention_f32(const AttentionF32& p, cudaStream_t s) {
    const size_t smem = sizeof(float) * ((size_t)(AF_STAGES * AF_SUB + AF_ROWS) * (p.d + 4) + AF_ROWS * AF_LDS);
    const int tiles = (p.n_tokens + AF_ROWS - 1) / AF_ROWS;
    // the runs of a tile go to one block each while the launch has few blocks (a decode step of 64 requests and 32 heads: 2048
    // runs), to fewer the more tiles there are (most blocks of a prompt's tiles would find no run)
    const long long want = 16LL * st_sm_count(), have = (long long)tiles * p.nh;
    int z = (int)((want + have - 1) / have);
    z = z > AF_ROWS ? AF_ROWS : z;
    if (z > p.n_tokens) z = p.n_tokens;
    if (have > 0x7fffffffLL) return ST_ERR_TOO_LARGE;
    dim3 grid((unsigned)have, 1, z);
    if (af_few(p)) {
        const size_t few = sizeof(float) * (2 * AF_SUB * p.d + p.d + KT);
        const cudaError_t e = cudaFuncSetAttribute(attention_f32_few_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)few);
        if (e != cudaSuccess) return (int)e;
        attention_f32_few_kernel<<<p.n_tokens * p.nh, KT, few, s>>>(p);
        return st_launch_status();
    }
#define AF_LAUNCH(NI)                                                                                                  \
    do {                                                                                                               \
        const cudaError_t e = cudaFuncSetAttribute(attention_f32_kernel<NI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
        if (e != cudaSuccess) return (int)e;                                                                           \
        attention_f32_kernel<NI><<<grid, KT, smem, s>>>(p);                                                            \
    } while (0)
    if (p.d <= 64) AF_LAUNCH(1);
    else if (p.d <= 128) AF_LAUNCH(2);
    else AF_LAUNCH(4);
#undef AF_LAUNCH
    return st_launch_status();
}

ST_EXPORT int st_attention_plain(const void* q, const void* pool, void* out, const int* positions,
                                 const int* seq_of_token, const int* slots, const int* block_table, int max_pages,
                                 int n_layers, int layer, int n_tokens, int nh, int nkv, int d, int page_size,
                                 float scale, int window, int dtype, int* status, void* stream, int n_seqs) {
    if (n_tokens <= 0) return 0;
    if (nh <= 0 || nkv <= 0 || nh % nkv || d <= 0 || page_size <= 0) return ST_ERR_BAD_ARG;
    if (d > 2 * KT) return ST_ERR_TOO_LARGE;
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == 0 && d % 4 == 0 && aligned16(q) && aligned16(pool) && aligned16(out) && nh <= 65535)
        return attention_f32({(const float*)q, (const float*)pool, (float*)out, positions, seq_of_token, slots, block_table,
                              n_tokens, max_pages, n_layers, layer, nh, nkv, d, page_size, window, scale, status, n_seqs}, s);
    dim3 grid(n_tokens, nh);
    const size_t smem = (size_t)(d + KT) * sizeof(float);
    if (dtype == 0)
        attention_plain_kernel<float><<<grid, KT, smem, s>>>((const float*)q, (const float*)pool, (float*)out,
            positions, seq_of_token, slots, block_table, max_pages, n_layers, layer, nh, nkv, d, page_size, scale, window, status);
    else if (dtype == 1)
        attention_plain_kernel<bf16><<<grid, KT, smem, s>>>((const bf16*)q, (const bf16*)pool, (bf16*)out,
            positions, seq_of_token, slots, block_table, max_pages, n_layers, layer, nh, nkv, d, page_size, scale, window, status);
    else return ST_ERR_BAD_DTYPE;
    return st_launch_status();
}
