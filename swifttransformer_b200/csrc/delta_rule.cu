// The gated delta rule: a linear recurrence whose state is corrected towards each token's value.
//
// Per value head h (G query/key heads serve H value heads: g = h / (H / G)), with S [dim, vd] zero when a
// request starts:
//
//   q, k, v  = silu(conv(projection))            short causal convolution over time, one filter per channel
//   q <- q / sqrt(sum q^2 + 1e-6) * dim^(-1/2),  k <- k / sqrt(sum k^2 + 1e-6)          per head
//   beta     = sigmoid(b)                                                              per head
//   decay_c  = exp(-exp(A_log_h) * softplus(sum_r a1_r * W_a2[h * dim + c, r] + dt_bias[h * dim + c]))
//   S <- diag(decay) S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
//   out      = out_scale * o / sqrt(mean(o^2) + eps) * w * sigmoid(sum_r g1_r * W_g2[h * vd + e, r])
//
// Two simpler forms of the same are taken by rank: with rank_a == 0 the projection holds one decay logit per head
// at a_off (dt_bias is then [H] and all key channels of a head decay alike); with rank_g == 0 it holds the output
// gate's logits themselves at g_off ([H * vd]).  gate_silu: the gate is z * sigmoid(z) instead of sigmoid(z).
//
// Three kernels.  delta_prepare turns a token's row of the float projection [q | k | v | b | a1 | g1] into a
// float row [q (G*dim) | k (G*dim) | v (H*vd) | decay (H*dim) | beta (H)]; delta_scan walks each request's
// tokens with the state's columns in registers (a column of S evolves on its own: its dot products with k and q
// are sums over dim, shared by the L lanes that hold the column) and the tokens' rows staged in shared memory; delta_output norms and gates each head's o.
// Everything here is float arithmetic; only the low-rank matrices and the result are in the storage type.
//
// Since (decay S + k u^T)^T q = (decay S)^T q + u (k . q), both dot products of a token are taken from the
// decayed state in one pass of shuffles.
#include "chunks.cuh"
#include "delta_rule.cuh"

#define DR_MAX_TAPS 8
#define DR_PREP_THREADS 256
#define DR_EARLY_TOKENS 128   // steps of at most this many tokens let the next kernel's blocks in early
#define DR_UNIT_PASSES 8      // a warp's lanes cover a head of up to 32 * DR_UNIT_PASSES channels

__device__ __forceinline__ float softplusf_(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// sum_r x[r] * w[r] in the order of r, the weights fetched in 16-byte pieces where the row allows it
#define DR_RANK_SMEM 256      // low-rank inputs of up to this many numbers wait in shared memory
template <typename TW>
__device__ __forceinline__ float lowrank_dot(const float* x, const TW* __restrict__ w, int rank) {
    float z = 0.f;
    if constexpr (sizeof(TW) == 2) {
        if ((rank & 7) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0) {
            for (int r = 0; r < rank; r += 8) {
                const uint4 u = __ldg(reinterpret_cast<const uint4*>(w + r));
                const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    z = fmaf(x[r + 2 * i], __uint_as_float(w4[i] << 16), z);
                    z = fmaf(x[r + 2 * i + 1], __uint_as_float(w4[i] & 0xffff0000u), z);
                }
            }
            return z;
        }
    } else {
        if ((rank & 3) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0) {
            for (int r = 0; r < rank; r += 4) {
                const float4 u = __ldg(reinterpret_cast<const float4*>(w + r));
                z = fmaf(x[r], u.x, z); z = fmaf(x[r + 1], u.y, z); z = fmaf(x[r + 2], u.z, z); z = fmaf(x[r + 3], u.w, z);
            }
            return z;
        }
    }
    for (int r = 0; r < rank; ++r) z = fmaf(x[r], to_f32(w[r]), z);
    return z;
}

// conv_w: float [2*G*dim + H*vd, taps] in the projection's order q | k | v; state: [slots, taps-1, channels]
// float, the last taps-1 projected rows of every request (read here; with move_state, in steps where every request
// brings one token, also moved on here: the thread that reads a channel's state is the only one that writes it).
template <typename TW>
__global__ void __launch_bounds__(DR_PREP_THREADS)
delta_prepare_kernel(const float* __restrict__ proj, int ld, DeltaShape sh, const float* __restrict__ conv_w,
                     float* __restrict__ state, int move_state, int taps, const TW* __restrict__ w_a2,
                     const float* __restrict__ a_log, const float* __restrict__ dt_bias, float* __restrict__ prep,
                     const int* __restrict__ positions, const int* __restrict__ seq_of_token,
                     const int* __restrict__ q_start, const int* __restrict__ slots) {
    ST_PDL_WAIT();
    // In a step of few tokens the recurrence's blocks may come in at once.  In a long portion they come in when this
    // grid is all but done: let in early, they were placed on the few multiprocessors that had room beside this
    // grid's blocks, many to each, and the walk over 2048 tokens took nearly twice as long (measured).
    const bool early = gridDim.x <= DR_EARLY_TOKENS;
    if (early) ST_PDL_TRIGGER();
    const int t = blockIdx.x;
    const int pos = positions[t];
    if (pos < 0) return;
    const int b = seq_of_token[t];
    const int i = t - q_start[b];                         // the token's place in its portion
    const int H = sh.H, G = sh.G, dim = sh.dim, vd = sh.vd;
    const int channels = 2 * G * dim + H * vd;
    const int keep = taps - 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const float* row = proj + (size_t)t * ld;
    float* st = state + (size_t)slots[b] * keep * channels;
    float* dst = prep + (size_t)t * sh.stride;
    const int units = 2 * G + H;
    for (int u = blockIdx.y * nwarp + warp; u < units; u += nwarp * gridDim.y) {
        const bool is_v = u >= 2 * G;
        const int width = is_v ? vd : dim;
        const int ch0 = is_v ? 2 * G * dim + (u - 2 * G) * vd : u * dim;     // q heads, then k heads, then v heads
        float x[DR_UNIT_PASSES];
        float ss = 0.f;
#pragma unroll
        for (int r = 0; r < DR_UNIT_PASSES; ++r) {
            x[r] = 0.f;
            const int e = lane + 32 * r;
            if (e >= width) continue;
            const int c = ch0 + e;
            // the projection's columns q_off.. hold q | k | v in this order
            float y = 0.f, vv[DR_MAX_TAPS];
            for (int j = 0; j < taps; ++j) {
                const int back = keep - j;
                float v;
                if (back <= i) v = __ldcg(row - (size_t)back * ld + sh.q_off + c);
                else v = __ldcg(st + (size_t)(keep - (back - i)) * channels + c);    // zero before the request's start
                vv[j] = v;
                y = fmaf(conv_w[(size_t)c * taps + j], v, y);
            }
            if (move_state)
                for (int j = 0; j < keep; ++j) st[(size_t)j * channels + c] = vv[j + 1];
            y = hk_silu(y);
            x[r] = y;
            ss = fmaf(y, y, ss);
        }
        float mult = 1.f;
        if (!is_v) {
            ss = warp_sum(ss);
            mult = rsqrtf(ss + 1e-6f);
            if (u < G) mult *= rsqrtf((float)dim);
        }
#pragma unroll
        for (int r = 0; r < DR_UNIT_PASSES; ++r) {
            const int e = lane + 32 * r;
            if (e < width) dst[ch0 + e] = x[r] * mult;       // the prepared row starts with q | k | v as well
        }
    }
    if (blockIdx.y == 0) {
        for (int h = threadIdx.x; h < H; h += blockDim.x)
            dst[sh.pb() + h] = hk_sigmoid(__ldcg(row + sh.b_off + h));
    }
    // decays: the low-rank step size, one thread per (head, key channel)
    __shared__ float xs_a[DR_RANK_SMEM];
    const float* xa = row + sh.a_off;
    if (sh.rank_a > 0 && sh.rank_a <= DR_RANK_SMEM) {
        for (int r = threadIdx.x; r < sh.rank_a; r += blockDim.x) xs_a[r] = __ldcg(xa + r);
        __syncthreads();
        xa = xs_a;
    }
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < H * dim; c += blockDim.x * gridDim.y) {
        float z, bias;
        if (sh.rank_a > 0) {
            z = lowrank_dot(xa, w_a2 + (size_t)c * sh.rank_a, sh.rank_a);
            bias = dt_bias[c];
        } else {
            z = __ldcg(xa + c / dim);
            bias = dt_bias[c / dim];
        }
        const float dt = softplusf_(z + bias);
        dst[sh.pd() + c] = expf(-expf(a_log[c / dim]) * dt);
    }
    if (!early) ST_PDL_TRIGGER();
}

// ---- delta_prepare for steps of many tokens -------------------------------------------------------------------
// delta_prepare_kernel has every token fetch its filters, low-rank weights and past rows again, by 80 KB of code that a block runs
// once; here a warp takes one head of q, k or v and a thread one key channel's decay through `run` tokens in a row (at most DR_RUN): filters
// and weights stay in registers, a token's past rows are the registers of the tokens before.  Every sum is delta_prepare_kernel's in
// the same order: a token's numbers do not depend on who shares its step.
// us on one B200, 2000 tokens, 8 value heads and 4 key heads of 128, rank 16 (41 MB of rows): 21 where delta_prepare_kernel takes 56; with
// runs of eight or four tokens where sixteen would leave the SMs idle 1501 tokens of 4 heads are 10 us faster, with sixteen 7 slower.
// Bound by instructions: some 120 of each decay's, 50 of each channel's.
#define DR_RUN 16
#define DR_RUN_OUT 4
#define DR_RUN_LOW 64         // low-rank inputs (or heads, without the pair) per token kept in shared memory
#define DR_RUN_UNITS 4        // a lane's channels of a head of up to 128: lane, lane + 32, ..

// sixteen low-rank weights of a row (16-byte aligned)
__device__ __forceinline__ void dr_sixteen(const float* p, float* w) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(p) + i);
        w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
    }
}
__device__ __forceinline__ void dr_sixteen(const bf16* p, float* w) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const uint4 u = __ldg(reinterpret_cast<const uint4*>(p) + i);
        const uint32_t u4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            w[8 * i + 2 * j] = __uint_as_float(u4[j] << 16);
            w[8 * i + 2 * j + 1] = __uint_as_float(u4[j] & 0xffff0000u);
        }
    }
}

// RANK: 16, 0 (no pair) or -1 (any rank up to DR_RUN_LOW)
template <typename TW, int TAPS, int RANK>
__global__ void __launch_bounds__(DR_PREP_THREADS)
delta_prepare_run_kernel(const float* __restrict__ proj, int ld, DeltaShape sh, const float* __restrict__ conv_w,
                         const float* __restrict__ state, int conv_blocks, const TW* __restrict__ w_a2,
                         const float* __restrict__ a_log, const float* __restrict__ dt_bias, float* __restrict__ prep,
                         const int* __restrict__ positions, const int* __restrict__ seq_of_token,
                         const int* __restrict__ q_start, const int* __restrict__ slots, int n_tokens, int run) {
    constexpr int KEEP = TAPS - 1;
    __shared__ int s_place[DR_RUN], s_slot[DR_RUN];          // a token's place in its portion (-1: padding), its request's slot
    __shared__ __align__(16) float s_low[DR_RUN][DR_RUN_LOW];
    const int tid = threadIdx.x, lane = tid & 31, t0 = blockIdx.x * run, n_run = min(run, n_tokens - t0);
    const int H = sh.H, G = sh.G, dim = sh.dim, vd = sh.vd;
    ST_PDL_WAIT();
    if ((int)blockIdx.y < conv_blocks) {
        if (tid < n_run) {
            const int b = seq_of_token[t0 + tid];
            const bool on = positions[t0 + tid] >= 0;
            s_place[tid] = on ? t0 + tid - q_start[b] : -1;
            s_slot[tid] = on ? slots[b] : 0;
        }
        __syncthreads();
        const int u = blockIdx.y * (DR_PREP_THREADS / 32) + (tid >> 5), channels = 2 * G * dim + H * vd;
        const bool is_v = u >= 2 * G;
        const int width = is_v ? vd : dim;
        const int c = (is_v ? 2 * G * dim + (u - 2 * G) * vd : u * dim) + lane;
        if (u < 2 * G + H) {
            float w[DR_RUN_UNITS][TAPS], past[DR_RUN_UNITS][KEEP > 0 ? KEEP : 1];        // past: the rows 1 .. KEEP before the next token
#pragma unroll
            for (int r = 0; r < DR_RUN_UNITS; ++r)
#pragma unroll
                for (int j = 0; j < TAPS; ++j) w[r][j] = lane + 32 * r < width ? conv_w[(size_t)(c + 32 * r) * TAPS + j] : 0.f;
            const float* src = proj + (size_t)t0 * ld + sh.q_off + c;
            bool follows = false;                            // `past` belongs to the token at hand
#pragma unroll 1
            for (int g = 0; g < n_run; g += 4) {
                float v[4][DR_RUN_UNITS];
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (int r = 0; r < DR_RUN_UNITS; ++r)
                        v[k][r] = lane + 32 * r < width ? __ldcg(src + (size_t)min(g + k, n_run - 1) * ld + 32 * r) : 0.f;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int t = g + k, place = t < n_run ? s_place[t] : -1;
                    if (place < 0) { follows = false; continue; }
                    if (!follows || place == 0) {
                        const float* st = state + (size_t)s_slot[t] * KEEP * channels + c;
#pragma unroll
                        for (int back = 1; back <= KEEP; ++back)
#pragma unroll
                            for (int r = 0; r < DR_RUN_UNITS; ++r)
                                past[r][back - 1] = lane + 32 * r >= width ? 0.f
                                                    : back <= place ? __ldcg(src + ((long long)t - back) * ld + 32 * r)
                                                                    : __ldcg(st + (size_t)(KEEP - (back - place)) * channels + 32 * r);
                    }
                    follows = true;
                    float y[DR_RUN_UNITS], ss = 0.f;
#pragma unroll
                    for (int r = 0; r < DR_RUN_UNITS; ++r) {
                        y[r] = 0.f;
#pragma unroll
                        for (int back = KEEP; back >= 1; --back) y[r] = fmaf(w[r][KEEP - back], past[r][back - 1], y[r]);
                        y[r] = fmaf(w[r][KEEP], v[k][r], y[r]);
                        y[r] = hk_silu(y[r]);
                        if (lane + 32 * r < width) ss = fmaf(y[r], y[r], ss);
                    }
                    float mult = 1.f;
                    if (!is_v) {
                        ss = warp_sum(ss);
                        mult = rsqrtf(ss + 1e-6f);
                        if (u < G) mult *= rsqrtf((float)dim);
                    }
                    float* dst = prep + (size_t)(t0 + t) * sh.stride + c;
#pragma unroll
                    for (int r = 0; r < DR_RUN_UNITS; ++r) {
                        if (lane + 32 * r < width) dst[32 * r] = y[r] * mult;
#pragma unroll
                        for (int back = KEEP; back >= 2; --back) past[r][back - 1] = past[r][back - 2];
                        past[r][0] = v[k][r];
                    }
                }
            }
        }
    } else {
        if (tid < n_run) s_place[tid] = positions[t0 + tid];
        const int low = RANK == 0 ? H : sh.rank_a;
        for (int i = tid; i < n_run * DR_RUN_LOW; i += DR_PREP_THREADS) {
            const int t = i / DR_RUN_LOW, r = i % DR_RUN_LOW;
            if (r < low) s_low[t][r] = __ldcg(proj + (size_t)(t0 + t) * ld + sh.a_off + r);
        }
        __syncthreads();
        if ((int)blockIdx.y == conv_blocks)
            for (int i = tid; i < n_run * H; i += DR_PREP_THREADS) {
                const int t = i / H, h = i % H;
                if (s_place[t] >= 0)
                    prep[(size_t)(t0 + t) * sh.stride + sh.pb() + h] = hk_sigmoid(__ldcg(proj + (size_t)(t0 + t) * ld + sh.b_off + h));
            }
        const int c = (blockIdx.y - conv_blocks) * DR_PREP_THREADS + tid;
        if (c < H * dim) {
            const int h = c / dim;
            const float rate = expf(a_log[h]), bias = dt_bias[RANK == 0 ? h : c];
            float w[RANK > 0 ? RANK : 1];
            if constexpr (RANK > 0) dr_sixteen(w_a2 + (size_t)c * RANK, w);
            float* dst = prep + (size_t)t0 * sh.stride + sh.pd() + c;
#pragma unroll 4
            for (int t = 0; t < n_run; ++t) {
                float z = 0.f;
                if constexpr (RANK > 0) {
#pragma unroll
                    for (int r = 0; r < RANK; r += 4) {
                        const float4 x = load4(&s_low[t][r]);
                        z = fmaf(x.x, w[r], z); z = fmaf(x.y, w[r + 1], z); z = fmaf(x.z, w[r + 2], z); z = fmaf(x.w, w[r + 3], z);
                    }
                } else if constexpr (RANK == 0) {
                    z = s_low[t][h];
                } else {
                    z = lowrank_dot(s_low[t], w_a2 + (size_t)c * sh.rank_a, sh.rank_a);
                }
                if (s_place[t] >= 0) dst[(size_t)t * sh.stride] = expf(-rate * softplusf_(z + bias));
            }
        }
    }
    ST_PDL_TRIGGER();
}

// ------------------------------------------------------------------------------------------------
// The recurrence.  grid (requests of the step, H, column groups); a block of DS_THREADS threads holds
// DS_THREADS / L columns of one head's state, L lanes per column with R rows each (dim <= L * R); lane `sub` of a
// column holds rows sub * R .. sub * R + R - 1.
//
// A token's step is short (a few hundred cycles) and the next one cannot start before it ends, so a trip to
// memory per token would be most of the time.  The block therefore brings the prepared rows of DS_CHUNK tokens at
// a time into shared memory with asynchronous 4-byte copies, DS_STAGES chunks deep: per token the head's k, q and
// decays (dimension sub * R + r at r * L + sub, so that the lanes of a column read neighbouring banks and the
// columns of a warp the same word), the block's values and beta.  Every thread then reads its 3 R numbers of the
// next token from shared memory while this token's sums travel through the shuffles.
#define DS_THREADS 128
#define DS_CHUNK 8
#define DS_STAGES 3

__device__ __forceinline__ void cp_async4s(uint32_t dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src));
}
__device__ __forceinline__ void ds_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void ds_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

template <int L, int R>
struct DeltaScanSmem {
    static constexpr int COLS = DS_THREADS / L;
    static constexpr int DP = L * R;                     // padded key size
    static constexpr int ROW = 3 * DP + COLS + 1;        // k | q | decay | the block's values | beta
    static constexpr size_t BYTES = (size_t)DS_STAGES * DS_CHUNK * ROW * sizeof(float);
};

template <int L, int R>
__global__ void __launch_bounds__(DS_THREADS)
delta_scan_kernel(const float* __restrict__ prep, DeltaShape sh, float* __restrict__ state, int write_state,
                  float* __restrict__ o_out, const int* __restrict__ positions, const int* __restrict__ q_start,
                  const int* __restrict__ slots, int below) {
    using M = DeltaScanSmem<L, R>;
    extern __shared__ __align__(16) float ds_smem[];
    ST_PDL_WAIT();
    const int b = blockIdx.x, h = blockIdx.y;
    const int first = q_start[b], n = q_start[b + 1] - first;
    if (n <= 0 || n >= below || positions[first] < 0) return;      // padding of a fixed-shape step; longer ones run in chunks
    const int H = sh.H, dim = sh.dim, vd = sh.vd;
    const int g = h / (H / sh.G);
    const int sub = threadIdx.x % L;
    const int col0 = blockIdx.z * M::COLS;
    const int col = col0 + threadIdx.x / L;
    const bool live = col < vd;
    const int d0 = sub * R;
    float* S = state + (((size_t)slots[b] * H + h) * dim) * vd + col;
    float s[R];
#pragma unroll
    for (int r = 0; r < R; ++r) s[r] = (live && d0 + r < dim) ? S[(size_t)(d0 + r) * vd] : 0.f;
    const int row_len = sh.stride;
    const float* p = prep + (size_t)first * row_len;
    // the padding of the staged rows (dimensions past dim, columns past vd) stays zero: nothing is copied there
    for (int i = threadIdx.x; i < DS_STAGES * DS_CHUNK * M::ROW; i += DS_THREADS) ds_smem[i] = 0.f;
    __syncthreads();
    const int n_chunks = (n + DS_CHUNK - 1) / DS_CHUNK;
    // What this thread copies for every token is fixed for the launch: JN key dimensions (their k, q and decay) and
    // one of the block's values or beta.  The places are worked out once; per token a copy is then an addition.
    constexpr int JN = (M::DP + DS_THREADS - 1) / DS_THREADS;
    int src_k[JN], src_q[JN], src_d[JN];
    uint32_t dst_at[JN];
    const uint32_t smem0 = (uint32_t)__cvta_generic_to_shared(ds_smem);
#pragma unroll
    for (int ji = 0; ji < JN; ++ji) {
        const int j = threadIdx.x + ji * DS_THREADS;
        src_k[ji] = j < dim ? sh.pk() + g * dim + j : -1;
        src_q[ji] = sh.pq() + g * dim + j;
        src_d[ji] = sh.pd() + h * dim + j;
        dst_at[ji] = (uint32_t)((j % R) * L + j / R) * 4u;
    }
    int src_x = -1;                                        // the value of one of the block's columns, or beta
    if (threadIdx.x < M::COLS) {
        if (col0 + threadIdx.x < vd) src_x = sh.pv() + h * vd + col0 + threadIdx.x;
    } else if (threadIdx.x == M::COLS) {
        src_x = sh.pb() + h;
    }
    const uint32_t dst_x = (uint32_t)(3 * M::DP + threadIdx.x) * 4u;
    auto stage_chunk = [&](int c) {
        uint32_t dst = smem0 + (uint32_t)((c % DS_STAGES) * DS_CHUNK * M::ROW) * 4u;
        const int t_end = min(DS_CHUNK, n - c * DS_CHUNK);
        const float* row = p + (size_t)(c * DS_CHUNK) * row_len;
#pragma unroll
        for (int t = 0; t < DS_CHUNK; ++t) {
            if (t < t_end) {
#pragma unroll
                for (int ji = 0; ji < JN; ++ji) {
                    if (src_k[ji] >= 0) {
                        cp_async4s(dst + dst_at[ji], row + src_k[ji]);
                        cp_async4s(dst + (uint32_t)M::DP * 4u + dst_at[ji], row + src_q[ji]);
                        cp_async4s(dst + (uint32_t)M::DP * 8u + dst_at[ji], row + src_d[ji]);
                    }
                }
                if (src_x >= 0) cp_async4s(dst + dst_x, row + src_x);
            }
            row += row_len;
            dst += (uint32_t)M::ROW * 4u;
        }
    };
#pragma unroll
    for (int c = 0; c < DS_STAGES - 1; ++c) {
        if (c < n_chunks) stage_chunk(c);
        ds_commit();
    }
    float* o_at = o_out + (size_t)first * H * vd + h * vd + col;
    const size_t o_step = (size_t)H * vd;
    const bool writes_o = live && sub == 0;
    float kq[R], qq[R], dd[R], v, beta;
    auto fetch = [&](const float* row) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            kq[r] = row[r * L + sub];
            qq[r] = row[M::DP + r * L + sub];
            dd[r] = row[2 * M::DP + r * L + sub];
        }
        v = row[3 * M::DP + threadIdx.x / L];
        beta = row[3 * M::DP + M::COLS];
    };
    for (int c = 0; c < n_chunks; ++c) {
        ds_wait<DS_STAGES - 2>();           // chunk c has landed (this thread's copies; the barrier makes it all threads')
        __syncthreads();                    // also: every thread is done with chunk c - 1, whose stage is filled next
        if (c + DS_STAGES - 1 < n_chunks) stage_chunk(c + DS_STAGES - 1);
        ds_commit();
        const float* rows = ds_smem + (size_t)(c % DS_STAGES) * DS_CHUNK * M::ROW;
        const int t_end = min(DS_CHUNK, n - c * DS_CHUNK);
        fetch(rows);
        for (int t = 0; t < t_end; ++t) {
            float k_[R];
            // partial sums in four lanes of arithmetic, so that the chain of additions is R / 4 long
            float sk4[4] = {0.f, 0.f, 0.f, 0.f}, sq4[4] = {0.f, 0.f, 0.f, 0.f}, kq4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int r = 0; r < R; ++r) {
                k_[r] = kq[r];
                s[r] *= dd[r];
                sk4[r & 3] = fmaf(s[r], k_[r], sk4[r & 3]);
                sq4[r & 3] = fmaf(s[r], qq[r], sq4[r & 3]);
                kq4[r & 3] = fmaf(k_[r], qq[r], kq4[r & 3]);
            }
            float sk = (sk4[0] + sk4[1]) + (sk4[2] + sk4[3]);
            float sq = (sq4[0] + sq4[1]) + (sq4[2] + sq4[3]);
            float kdq = (kq4[0] + kq4[1]) + (kq4[2] + kq4[3]);
            const float v_now = v, beta_now = beta;
            if (t + 1 < t_end) fetch(rows + (t + 1) * M::ROW);      // the next token's numbers are on their way meanwhile
#pragma unroll
            for (int o = L / 2; o > 0; o >>= 1) {
                sk += __shfl_xor_sync(0xffffffffu, sk, o);
                sq += __shfl_xor_sync(0xffffffffu, sq, o);
                kdq += __shfl_xor_sync(0xffffffffu, kdq, o);
            }
            const float u = beta_now * (v_now - sk);
#pragma unroll
            for (int r = 0; r < R; ++r) s[r] = fmaf(k_[r], u, s[r]);
            if (writes_o) *o_at = fmaf(u, kdq, sq);
            o_at += o_step;
        }
    }
    // The successor's blocks are let in only now: while they wait for this grid on the same multiprocessors, the
    // walk over a long portion was measured to take nearly twice as long.
    ST_PDL_TRIGGER();
    ds_wait<0>();
    if (write_state && live) {
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (d0 + r < dim) S[(size_t)(d0 + r) * vd] = s[r];
    }
}

// out[t, h, e] = out_scale * o / sqrt(mean_e o^2 + eps) * norm_w[e] * sigmoid(sum_r g1[t, r] * W_g2[h * vd + e, r])
template <typename T>
__global__ void __launch_bounds__(128)
delta_output_kernel(const float* __restrict__ o, const float* __restrict__ proj, int ld, DeltaShape sh,
                    const T* __restrict__ w_g2, const float* __restrict__ norm_w, float eps, float out_scale,
                    T* __restrict__ out, const int* __restrict__ positions) {
    __shared__ float scratch[32];
    ST_PDL_WAIT();
    ST_PDL_TRIGGER();
    const int t = blockIdx.x, h = blockIdx.y;
    if (positions[t] < 0) return;
    const int vd = sh.vd;
    const float* orow = o + ((size_t)t * sh.H + h) * vd;
    float ss = 0.f;
    for (int e = threadIdx.x; e < vd; e += blockDim.x) {
        const float x = __ldcg(orow + e);
        ss = fmaf(x, x, ss);
    }
    ss = block_sum(ss, scratch);
    const float inv = rsqrtf(ss / (float)vd + eps) * out_scale;
    __shared__ float xs_g[DR_RANK_SMEM];
    const float* g1 = proj + (size_t)t * ld + sh.g_off;
    if (sh.rank_g > 0 && sh.rank_g <= DR_RANK_SMEM) {
        for (int r = threadIdx.x; r < sh.rank_g; r += blockDim.x) xs_g[r] = __ldcg(g1 + r);
        __syncthreads();
        g1 = xs_g;
    }
    for (int e = threadIdx.x; e < vd; e += blockDim.x) {
        const float z = sh.rank_g > 0 ? lowrank_dot(g1, w_g2 + (size_t)(h * vd + e) * sh.rank_g, sh.rank_g)
                                      : __ldcg(g1 + h * vd + e);
        const float gate = sh.gate_silu ? hk_silu(z) : hk_sigmoid(z);
        out[((size_t)t * sh.H + h) * vd + e] = from_f32<T>(__ldcg(orow + e) * inv * norm_w[e] * gate);
    }
}

// delta_output for steps of many tokens: a warp takes a head through DR_RUN_OUT tokens, the low-rank weights in registers; its sums are
// delta_output_kernel's in the same order.  15 us where that takes 24 (2000 tokens, 8 heads of 128, rank 16); sixteen tokens a warp, 34
template <typename T, int RANK>
__global__ void __launch_bounds__(DR_PREP_THREADS)
delta_output_run_kernel(const float* __restrict__ o, const float* __restrict__ proj, int ld, DeltaShape sh, const T* __restrict__ w_g2,
                        const float* __restrict__ norm_w, float eps, float out_scale, T* __restrict__ out,
                        const int* __restrict__ positions, int n_tokens) {
    __shared__ __align__(16) float s_low[DR_RUN_OUT][DR_RUN_LOW];
    __shared__ int s_on[DR_RUN_OUT];
    const int tid = threadIdx.x, lane = tid & 31, t0 = blockIdx.x * DR_RUN_OUT, n_run = min(DR_RUN_OUT, n_tokens - t0);
    const int h = blockIdx.y * (DR_PREP_THREADS / 32) + (tid >> 5), vd = sh.vd;
    float w[DR_RUN_UNITS][RANK > 0 ? RANK : 1], nw[DR_RUN_UNITS];
    bool on[DR_RUN_UNITS];
#pragma unroll
    for (int x = 0; x < DR_RUN_UNITS; ++x) {               // (weights: no kernel writes them)
        const int e = lane + 32 * x;
        on[x] = h < sh.H && e < vd;
        nw[x] = on[x] ? norm_w[e] : 0.f;
        if constexpr (RANK > 0)
            if (on[x]) dr_sixteen(w_g2 + ((size_t)h * vd + e) * RANK, w[x]);
    }
    ST_PDL_WAIT();
    ST_PDL_TRIGGER();
    if (tid < n_run) s_on[tid] = positions[t0 + tid] >= 0;
    if (RANK != 0)
        for (int i = tid; i < DR_RUN_OUT * DR_RUN_LOW; i += DR_PREP_THREADS) {
            const int t = i / DR_RUN_LOW, r = i % DR_RUN_LOW;
            if (t < n_run && r < sh.rank_g) s_low[t][r] = __ldcg(proj + (size_t)(t0 + t) * ld + sh.g_off + r);
        }
    float v[DR_RUN_OUT][DR_RUN_UNITS];
#pragma unroll
    for (int k = 0; k < DR_RUN_OUT; ++k)
#pragma unroll
        for (int x = 0; x < DR_RUN_UNITS; ++x)
            v[k][x] = on[x] ? __ldcg(o + ((size_t)(t0 + min(k, n_run - 1)) * sh.H + h) * vd + lane + 32 * x) : 0.f;
    __syncthreads();
    if (h >= sh.H) return;
#pragma unroll
    for (int k = 0; k < DR_RUN_OUT; ++k) {
        if (k >= n_run || !s_on[k]) continue;
        float ss = 0.f;
#pragma unroll
        for (int x = 0; x < DR_RUN_UNITS; ++x) ss += warp_sum(v[k][x] * v[k][x]);
        const float inv = rsqrtf(ss / (float)vd + eps) * out_scale;
#pragma unroll
        for (int x = 0; x < DR_RUN_UNITS; ++x) {
            if (!on[x]) continue;
            const int e = lane + 32 * x;
            float z = 0.f;
            if constexpr (RANK > 0) {
#pragma unroll
                for (int r = 0; r < RANK; r += 4) {
                    const float4 low = load4(&s_low[k][r]);
                    z = fmaf(low.x, w[x][r], z); z = fmaf(low.y, w[x][r + 1], z);
                    z = fmaf(low.z, w[x][r + 2], z); z = fmaf(low.w, w[x][r + 3], z);
                }
            } else if constexpr (RANK == 0) {
                z = __ldcg(proj + (size_t)(t0 + k) * ld + sh.g_off + h * vd + e);
            } else {
                z = lowrank_dot(s_low[k], w_g2 + ((size_t)h * vd + e) * sh.rank_g, sh.rank_g);
            }
            const float gate = sh.gate_silu ? hk_silu(z) : hk_sigmoid(z);
            out[((size_t)(t0 + k) * sh.H + h) * vd + e] = from_f32<T>(v[k][x] * inv * nw[x] * gate);
        }
    }
}

// 0: the launcher chooses the lanes per column of the recurrence; 8 or 16: this many (for tests and tuning).
static int ds_forced_lanes = 0;
ST_EXPORT int st_delta_rule_set_lanes(int lanes) {
    if (lanes != 0 && lanes != 8 && lanes != 16) return ST_ERR_BAD_ARG;
    ds_forced_lanes = lanes;
    return 0;
}
// Floats of scratch with which n_seqs requests of a step of n_tokens tokens run in chunks (0: they do not).
ST_EXPORT long long st_delta_rule_chunk_floats(int n_tokens, int n_seqs, int H, int G, int dim, int vd) {
    if (n_tokens <= 0 || n_seqs <= 0 || H <= 0 || G <= 0 || H % G || dim <= 0 || vd <= 0 || ds_forced_lanes) return 0;
    DeltaShape sh = {};
    sh.H = H; sh.G = G; sh.dim = dim; sh.vd = vd;
    const long long more = delta_chunks_floats(n_tokens, n_seqs, sh);
    return more ? (long long)n_tokens * ((sh.row() + 3) / 4 * 4 + (long long)H * vd) + more : 0;
}
// Floats of scratch for the walk.
ST_EXPORT long long st_delta_rule_scratch_floats(int n_tokens, int H, int G, int dim, int vd) {
    return (long long)n_tokens * ((long long)2 * G * dim + (long long)H * vd + (long long)H * dim + H + (long long)H * vd);
}

// proj: float [n_tokens, ld]; w_a2 [H*dim, rank_a], w_g2 [H*vd, rank_g] in the storage type `dtype`, as is out
// [n_tokens, H*vd]; conv_state float [slots, taps-1, 2*G*dim + H*vd]; state float [slots, H, dim, vd];
// scratch: float, st_delta_rule_scratch_floats elements.  write_state == 0: the states are read, not moved on.  from > 0: requests
// of at least so many tokens run in chunks (scratch: 16-byte aligned, st_delta_rule_chunk_floats elements for min(n_seqs,
// n_tokens / from) requests); walk == 0: there are no others.
ST_EXPORT int st_delta_rule(const float* proj, int ld, int q_off, int b_off, int a_off, int g_off, int rank_a,
                            int rank_g, const float* conv_w, int taps, float* conv_state, const void* w_a2,
                            const float* a_log, const float* dt_bias, const void* w_g2, const float* norm_w, float eps,
                            float out_scale, float* state, int write_state, int single_tokens, float* scratch,
                            void* out, const int* positions, const int* seq_of_token, const int* q_start,
                            const int* slots, int n_tokens, int n_seqs, int H, int G, int dim, int vd, int dtype,
                            void* stream, int gate_silu, int from, int walk) {
    if (n_tokens <= 0 || n_seqs <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || dim <= 0 || vd <= 0 || taps < 1 || rank_a < 0 || rank_g < 0) return ST_ERR_BAD_ARG;
    if (taps > DR_MAX_TAPS || dim > 32 * DR_UNIT_PASSES || vd > 32 * DR_UNIT_PASSES) return ST_ERR_TOO_LARGE;
    if (dtype != 0 && dtype != 1) return ST_ERR_BAD_DTYPE;
    DeltaShape sh;
    sh.H = H; sh.G = G; sh.dim = dim; sh.vd = vd;
    sh.q_off = q_off; sh.k_off = q_off + G * dim; sh.v_off = q_off + 2 * G * dim;
    sh.b_off = b_off; sh.a_off = a_off; sh.g_off = g_off; sh.rank_a = rank_a; sh.rank_g = rank_g; sh.gate_silu = gate_silu;
    if (from < 0 || (from == 0 && !walk)) return ST_ERR_BAD_ARG;
    const bool chunks = from > 0 && from <= n_tokens;
    const int below = chunks ? from : n_tokens + 1;
    sh.stride = chunks ? (sh.row() + 3) / 4 * 4 : sh.row();
    if (chunks && delta_chunks_floats(n_tokens, n_seqs, sh) == 0) return ST_ERR_BAD_SIZE;
    if (chunks && !aligned16(scratch)) return ST_ERR_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    float* prep = scratch;
    float* o = scratch + (size_t)n_tokens * sh.stride;
    const int move = single_tokens && write_state && taps > 1;
    int rc;
    // Which form of prepare and output: by runs of tokens where a step has enough of them to fill the multiprocessors, heads fit a
    // warp's registers and the tails are not moved on here
    const bool runs = n_tokens > DR_EARLY_TOKENS && !move && taps >= 2 && taps <= 4 && dim <= 32 * DR_RUN_UNITS && vd <= 32 * DR_RUN_UNITS &&
                      H <= DR_RUN_LOW && rank_a <= DR_RUN_LOW && rank_g <= DR_RUN_LOW;
    const bool sixteen_a = rank_a == 16 && aligned16(w_a2), sixteen_g = rank_g == 16 && aligned16(w_g2);
    if (runs) {
        const int conv_blocks = (2 * G + H + DR_PREP_THREADS / 32 - 1) / (DR_PREP_THREADS / 32);
        // sixteen tokens a run where that still gives four blocks per SM, else eight or four
        const int gy = conv_blocks + (H * dim + DR_PREP_THREADS - 1) / DR_PREP_THREADS;
        int run = DR_RUN;
        while (run > 4 && (long long)((n_tokens + run - 1) / run) * gy < 4 * st_sm_count()) run /= 2;
        const dim3 grid((unsigned)((n_tokens + run - 1) / run), gy);
#define DR_RUN_PREP(TW, TAPS, RANK)                                                                                   \
    rc = st_launch_pdl("delta_prepare", delta_prepare_run_kernel<TW, TAPS, RANK>, grid, dim3(DR_PREP_THREADS), 0, s, proj, ld, sh, conv_w, \
                       (const float*)conv_state, conv_blocks, (const TW*)w_a2, a_log, dt_bias, prep, positions, seq_of_token, q_start, \
                       slots, n_tokens, run)
#define DR_RUN_RANK(TW, TAPS)                                                                                         \
    do {                                                                                                              \
        if (sixteen_a) DR_RUN_PREP(TW, TAPS, 16);                                                                     \
        else if (rank_a == 0) DR_RUN_PREP(TW, TAPS, 0);                                                               \
        else DR_RUN_PREP(TW, TAPS, -1);                                                                               \
    } while (0)
#define DR_RUN_TAPS(TW)                                                                                               \
    do {                                                                                                              \
        if (taps == 4) DR_RUN_RANK(TW, 4);                                                                            \
        else if (taps == 3) DR_RUN_RANK(TW, 3);                                                                       \
        else DR_RUN_RANK(TW, 2);                                                                                      \
    } while (0)
        if (dtype == 0) DR_RUN_TAPS(float);
        else DR_RUN_TAPS(bf16);
#undef DR_RUN_TAPS
#undef DR_RUN_RANK
#undef DR_RUN_PREP
        if (rc) return rc;
    } else {
        const int units = 2 * G + H;
        int gy = (units + 7) / 8;
        if (gy > 16) gy = 16;
        dim3 grid(n_tokens, gy);
        if (dtype == 0)
            rc = st_launch_pdl("delta_prepare", delta_prepare_kernel<float>, grid, dim3(DR_PREP_THREADS), 0, s, proj, ld, sh,
                               conv_w, conv_state, move, taps, (const float*)w_a2, a_log, dt_bias, prep, positions,
                               seq_of_token, q_start, slots);
        else
            rc = st_launch_pdl("delta_prepare", delta_prepare_kernel<bf16>, grid, dim3(DR_PREP_THREADS), 0, s, proj, ld, sh,
                               conv_w, conv_state, move, taps, (const bf16*)w_a2, a_log, dt_bias, prep, positions,
                               seq_of_token, q_start, slots);
        if (rc) return rc;
    }
    if (!chunks || walk) {
#define DS_LAUNCH(L, R)                                                                                              \
    do {                                                                                                             \
        const size_t smem = DeltaScanSmem<L, R>::BYTES;                                                              \
        if (smem > 48 * 1024) {                                                                                      \
            cudaError_t e = cudaFuncSetAttribute(delta_scan_kernel<L, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                                 (int)smem);                                                         \
            if (e != cudaSuccess) return (int)e;                                                                     \
        }                                                                                                            \
        rc = st_launch_pdl("delta_scan", delta_scan_kernel<L, R>,                                                    \
                           dim3(n_seqs, H, (vd + DS_THREADS / L - 1) / (DS_THREADS / L)), dim3(DS_THREADS), smem, s, \
                           (const float*)prep, sh, state, write_state, o, positions, q_start, slots, below);         \
    } while (0)
        // Lanes per column.  A token's step is a chain of dependent instructions, so a launch is as fast as its
        // blocks are spread: when eight lanes per column give fewer blocks than the device has multiprocessors,
        // sixteen (fewer rows each, one more stage of shuffles) were measured faster, by a fifth for one request of
        // eight heads; for short columns (dim <= 32) and for steps of many requests eight are.  Thirty-two lanes
        // were measured too and never won.
        int lanes = ds_forced_lanes;
        if (!lanes) {
            const long long cols8 = (vd + DS_THREADS / 8 - 1) / (DS_THREADS / 8);
            lanes = (dim > 32 && (long long)n_seqs * H * cols8 < st_sm_count()) ? 16 : 8;
        }
        if (dim > 128) lanes = 16;
        if (lanes == 8) {
            if (dim <= 32) DS_LAUNCH(8, 4);
            else if (dim <= 64) DS_LAUNCH(8, 8);
            else DS_LAUNCH(8, 16);
        } else {
            if (dim <= 32) DS_LAUNCH(16, 2);
            else if (dim <= 64) DS_LAUNCH(16, 4);
            else if (dim <= 128) DS_LAUNCH(16, 8);
            else DS_LAUNCH(16, 16);
        }
#undef DS_LAUNCH
        if (rc) return rc;
    }
    if (chunks) {
        rc = delta_chunks_launch(prep, sh, o + (size_t)n_tokens * H * vd, state, write_state, o, positions, q_start, slots, n_tokens,
                                 n_seqs, from, s);
        if (rc) return rc;
    }
    if (runs) {
        const dim3 grid((unsigned)((n_tokens + DR_RUN_OUT - 1) / DR_RUN_OUT), (H + DR_PREP_THREADS / 32 - 1) / (DR_PREP_THREADS / 32));
#define DR_RUN_OUTPUT(T, RANK)                                                                                           \
    return st_launch_pdl("delta_output", delta_output_run_kernel<T, RANK>, grid, dim3(DR_PREP_THREADS), 0, s, (const float*)o, proj, ld, sh, \
                         (const T*)w_g2, norm_w, eps, out_scale, (T*)out, positions, n_tokens)
#define DR_RUN_RANK(T)                                                                                                \
    do {                                                                                                              \
        if (sixteen_g) DR_RUN_OUTPUT(T, 16);                                                                          \
        if (rank_g == 0) DR_RUN_OUTPUT(T, 0);                                                                            \
        DR_RUN_OUTPUT(T, -1);                                                                                            \
    } while (0)
        if (dtype == 0) DR_RUN_RANK(float);
        DR_RUN_RANK(bf16);
#undef DR_RUN_RANK
#undef DR_RUN_OUTPUT
    }
    dim3 grid(n_tokens, H);
    if (dtype == 0)
        return st_launch_pdl("delta_output", delta_output_kernel<float>, grid, dim3(128), 0, s, (const float*)o, proj, ld, sh,
                             (const float*)w_g2, norm_w, eps, out_scale, (float*)out, positions);
    return st_launch_pdl("delta_output", delta_output_kernel<bf16>, grid, dim3(128), 0, s, (const float*)o, proj, ld, sh,
                         (const bf16*)w_g2, norm_w, eps, out_scale, (bf16*)out, positions);
}
