// The gated delta rule of delta_rule.cu over long portions, in chunks of 64 tokens side by side.
//
//   S_t = D_t S_{t-1} + k_t u_t^T,   u_t = beta_t (v_t - (D_t S_{t-1})^T k_t),   o_t = S_t^T q_t        D_t = diag(decay_t)
//
// Walking the tokens is a chain of a few hundred clocks per token.  Over a chunk of C tokens after a state S, with the
// decays' products D(s, t) = D_{s+1} .. D_t, the u of the chunk solve a unit triangular system,
//
//   u_t + beta_t sum_{s < t} M[t][s] u_s = beta_t (v_t - S^T D(0, t) k_t),      M[t][s] = k_t^T D(s, t) k_s
//
// whose right side is linear in S: U = U0 - W S, where row t of U0 and W solve it for beta v and beta D(0, t) k.  Then
//
//   S_end = D(0, C) S + sum_s (D(s, C) k_s) u_s^T,      o_t = S^T (D(0, t) q_t) + sum_{s <= t} (q_t^T D(s, t) k_s) u_s
//
// (the representation of products of Householder-like factors by two tall matrices; Bischof and Van Loan 1987).  Three
// kernels between delta_prepare and delta_output: delta_chunk_prepare forms W, U0, the decayed q and k and the matrix of
// q^T D k of every chunk side by side; delta_chunk_walk carries the state from chunk to chunk, a block per head and 8 or 16
// of its value columns, as two products per chunk, and leaves U and the state before every chunk; delta_chunk_out forms the
// outputs.  All of it is float arithmetic, and every factor is a product of decays (at most 1), none a quotient.
//
// Measured on one B200, the whole operation with delta_prepare (56 us) and delta_output (24): 2000 tokens of one request, 8
// heads of 128 x 128, 283 us (prepare 55, walk 113, out 30) against 673 for the walk token by token (delta_scan 584); 16 heads
// 496 / 892; 500 tokens of 8 heads 126 / 194; 300: 119 / 138; 200: 100 / 93, so portions of fewer than 256 tokens stay with
// the walk.  Errors against 64 bits: outputs 2.24e-7 (walk 2.33e-7), states 3.34e-7 (3.67e-7).
#include "chunks.cuh"
#include "delta_rule.cuh"

struct ChunkScratch {
    float *W, *U, *Q, *K, *A, *P, *S;      // per (place, head): [64][dim], [64][vd], [64][dim], [64][dim], [64][64], [dim], [dim][vd]
};

// element (t, e) of the unpadded rows of delta_chunk_prepare: pieces of four turned by the row, so that reads of one piece of
// eight rows hit distinct banks
__device__ __forceinline__ int dc_at(int t, int e) { return t * HK_D + (e ^ ((t & 7) << 2)); }

struct DcPrepareSmem {
    float Q[HK_C * HK_D], K[HK_C * HK_D], F[HK_C * HK_D], AM[HK_C * HK_C], total[2][HK_D];
};

// AM holds q_t^T D(s, t) k_s at [t][s], s <= t, and k_t^T D(s, t) k_s at [s][t], s < t.
__global__ void __launch_bounds__(256, 2)
delta_chunk_prepare_kernel(const float* __restrict__ prep, const DeltaShape sh, const ChunkScratch cs,
                           const int* __restrict__ positions, const int* __restrict__ q_start, int n_seqs, int from) {
    extern __shared__ __align__(16) unsigned char dc_raw[];
    DcPrepareSmem& m = *reinterpret_cast<DcPrepareSmem*>(dc_raw);
    ST_PDL_WAIT();
    const int place = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int dim = sh.dim, vd = sh.vd, g = h / (sh.H / sh.G);
    int b, first, n;
    if (!hk_find(q_start, positions, n_seqs, from, place, b, first, n)) return;
    const size_t unit = (size_t)place * sh.H + h;
    const float* rows = prep + (size_t)first * sh.stride;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f), one = make_float4(1.f, 1.f, 1.f, 1.f);
    const float beta = tid < HK_C && tid < n ? __ldcg(rows + (size_t)tid * sh.stride + sh.pb() + h) : 0.f;
    const int e4 = (tid & 31) * 4, t8 = tid >> 5;           // a thread's pieces: four columns of every eighth row
    {
        float4 q[8], k[8], f[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float* row = rows + (size_t)min(t8 + 8 * i, n - 1) * sh.stride;
            const bool on = e4 < dim && t8 + 8 * i < n;
            q[i] = on ? load4_cg(row + sh.pq() + g * dim + e4) : zero;
            k[i] = on ? load4_cg(row + sh.pk() + g * dim + e4) : zero;
            f[i] = on ? load4_cg(row + sh.pd() + h * dim + e4) : one;
        }
        for (int i = tid; i < HK_C * HK_C / 4; i += 256) store4(m.AM + 4 * i, zero);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int at = dc_at(t8 + 8 * i, e4);
            store4(m.Q + at, q[i]);
            store4(m.K + at, k[i]);
            store4(m.F + at, f[i]);
        }
    }
    __syncthreads();
    for (int half = 0; half < HK_C; half += HK_H) {
        if (half >= n) break;
        // inside a half: a warp takes four s of it, its lanes four channels each; d[k] = D(s, t) k_s
        const int s_of[4] = {warp, 15 - warp, 16 + warp, 31 - warp};
        float4 d[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) d[k] = zero;
        const bool up16 = lane & 16, up8 = lane & 8, up4 = lane & 4;
        const int mine = up8 ? (up4 ? s_of[3] : s_of[2]) : (up4 ? s_of[1] : s_of[0]);
        const int t_end = min(HK_H, n - half);
#pragma unroll 2
        for (int t = 0; t < t_end; ++t) {
            const int at = dc_at(half + t, lane * 4);
            const float4 q = load4(m.Q + at), kt = load4(m.K + at), f = load4(m.F + at);
            float v[8];                                    // the four q sums, then the four k sums
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (t == s_of[k]) d[k] = kt;
                else d[k] = make_float4(d[k].x * f.x, d[k].y * f.y, d[k].z * f.z, d[k].w * f.w);
                v[k] = fmaf(q.x, d[k].x, fmaf(q.y, d[k].y, fmaf(q.z, d[k].z, q.w * d[k].w)));
                v[4 + k] = fmaf(kt.x, d[k].x, fmaf(kt.y, d[k].y, fmaf(kt.z, d[k].z, kt.w * d[k].w)));
            }
            // eight sums over 32 lanes: halves of the warp pass on the four they do not keep, then two, then one
            float w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) w[k] = (up16 ? v[4 + k] : v[k]) + __shfl_xor_sync(0xffffffffu, up16 ? v[k] : v[4 + k], 16);
            float x[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) x[k] = (up8 ? w[2 + k] : w[k]) + __shfl_xor_sync(0xffffffffu, up8 ? w[k] : w[2 + k], 8);
            float y = (up4 ? x[1] : x[0]) + __shfl_xor_sync(0xffffffffu, up4 ? x[0] : x[1], 4);
            y += __shfl_xor_sync(0xffffffffu, y, 2);
            y += __shfl_xor_sync(0xffffffffu, y, 1);
            if ((lane & 3) == 0) {
                if (!up16 && mine <= t) m.AM[(half + t) * HK_C + half + mine] = y;
                if (up16 && mine < t) m.AM[(half + mine) * HK_C + half + t] = y;
            }
        }
    }
    __syncthreads();
    {   // q and k decayed from their half's start (in Q and K), k decayed to its end (in F); read before overwritten.  The
        // products run over groups of eight and then over the groups: twelve roundings at most, not 32
        const int half = tid / HK_D, c = tid & (HK_D - 1), r0 = half * HK_H;
        float f[HK_H], k[HK_H], before = 1.f;
#pragma unroll
        for (int t = 0; t < HK_H; ++t) { f[t] = m.F[dc_at(r0 + t, c)]; k[t] = m.K[dc_at(r0 + t, c)]; }
#pragma unroll
        for (int t0 = 0; t0 < HK_H; t0 += 8) {
            float q[8], r = 1.f;
#pragma unroll
            for (int t = 0; t < 8; ++t) q[t] = m.Q[dc_at(r0 + t0 + t, c)];
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                r *= f[t0 + t];
                const float p = r * before;
                m.Q[dc_at(r0 + t0 + t, c)] = q[t] * p;
                m.K[dc_at(r0 + t0 + t, c)] = k[t0 + t] * p;
            }
            before *= r;
        }
        m.total[half][c] = before;
        float behind = 1.f;
#pragma unroll
        for (int t0 = HK_H - 8; t0 >= 0; t0 -= 8) {
            float r = 1.f;
#pragma unroll
            for (int t = 7; t >= 0; --t) {
                m.F[dc_at(r0 + t0 + t, c)] = k[t0 + t] * (r * behind);
                r *= f[t0 + t];
            }
            behind *= r;
        }
    }
    __syncthreads();
    if (n > HK_H) {                                         // between the halves: 2 x 2 sums of either kind per thread
        const int rl = (lane & 1) | ((lane >> 4) << 1), cl = (lane >> 1) & 7;
        const int t0 = HK_H + (warp >> 1) * 8 + rl, s0 = (warp & 1) * 16 + cl;
        float4 a[2][2], x[2][2];                            // four chains per sum
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i >> 1][i & 1] = x[i >> 1][i & 1] = zero;
#pragma unroll 2
        for (int e = 0; e < dim; e += 4) {
            float4 q[2], k[2], d[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                q[i] = load4(m.Q + dc_at(t0 + 4 * i, e));
                k[i] = load4(m.K + dc_at(t0 + 4 * i, e));
                d[i] = load4(m.F + dc_at(s0 + 8 * i, e));
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    a[i][j] = hk_fma4x4(q[i], d[j], a[i][j]);
                    x[i][j] = hk_fma4x4(k[i], d[j], x[i][j]);
                }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float4 y = a[i][j], z = x[i][j];
                m.AM[(t0 + 4 * i) * HK_C + s0 + 8 * j] = (y.x + y.y) + (y.z + y.w);
                m.AM[(s0 + 8 * j) * HK_C + t0 + 4 * i] = (z.x + z.y) + (z.z + z.w);
            }
    }
    __syncthreads();
    {   // the decayed q and k and A leave
        float* Qd = cs.Q + unit * HK_C * dim;
        float* Kd = cs.K + unit * HK_C * dim;
        float* A = cs.A + unit * HK_C * HK_C;
        if (e4 < dim) {
            const float4 w0 = load4(m.total[0] + e4), w1 = load4(m.total[1] + e4);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int t = t8 + 8 * i;
                float4 q = load4(m.Q + dc_at(t, e4)), k = load4(m.F + dc_at(t, e4));
                if (i >= 4) q = make_float4(q.x * w0.x, q.y * w0.y, q.z * w0.z, q.w * w0.w);
                else k = make_float4(k.x * w1.x, k.y * w1.y, k.z * w1.z, k.w * w1.w);
                store4(Qd + t * dim + e4, q);
                store4(Kd + t * dim + e4, k);
            }
            if (t8 == 0) store4(cs.P + unit * dim + e4, make_float4(w0.x * w1.x, w0.y * w1.y, w0.z * w1.z, w0.w * w1.w));
        }
        for (int i = tid; i < HK_C * HK_C / 4; i += 256) {
            const int t = i / (HK_C / 4), s = (i % (HK_C / 4)) * 4;
            const float4 v = load4(m.AM + 4 * i);
            store4(A + 4 * i, make_float4(s <= t ? v.x : 0.f, s + 1 <= t ? v.y : 0.f, s + 2 <= t ? v.z : 0.f, s + 3 <= t ? v.w : 0.f));
        }
    }
    float4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = t8 + 8 * i;
        v[i] = e4 < vd && t < n ? load4_cg(rows + (size_t)t * sh.stride + sh.pv() + h * vd + e4) : zero;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) store4(m.F + dc_at(t8 + 8 * i, e4), v[i]);      // the values take F's place,
    if (tid < HK_C) m.Q[tid] = beta;                                            // the write strengths Q's
    __syncthreads();
    {   // the triangular system, a thread per column: of D(0, t) k for W, of v for U0.  The corrections are summed up by
        // themselves and taken from the right side once (summed into it they cost a rounding of its size each)
        const bool for_w = tid < HK_D;
        const int c = tid & (HK_D - 1);
        if (c < (for_w ? dim : vd)) {
            const float* right = for_w ? m.K : m.F;
            const float w0 = for_w ? m.total[0][c] : 1.f;
            float* dst = for_w ? cs.W + unit * HK_C * dim + c : cs.U + unit * HK_C * vd + c;
            const int ld = for_w ? dim : vd;
            float y[HK_C];
#pragma unroll
            for (int t = 0; t < HK_C; ++t) y[t] = 0.f;
#pragma unroll
            for (int s = 0; s < HK_C; ++s) {
                const float x = m.Q[s] * (right[dc_at(s, c)] * (s >= HK_H ? w0 : 1.f) - y[s]);
                dst[s * ld] = x;
#pragma unroll
                for (int t = s / 4 * 4; t < HK_C; t += 4) {
                    if (t + 3 <= s) continue;
                    const float4 w = load4(m.AM + s * HK_C + t);
                    if (t > s) y[t] = fmaf(w.x, x, y[t]);
                    if (t + 1 > s) y[t + 1] = fmaf(w.y, x, y[t + 1]);
                    if (t + 2 > s) y[t + 2] = fmaf(w.z, x, y[t + 2]);
                    y[t + 3] = fmaf(w.w, x, y[t + 3]);
                }
            }
        }
    }
    ST_PDL_TRIGGER();
}

// ---- the state from chunk to chunk ------------------------------------------------------------------------------
// A block carries VS = 4 NC columns of a head's state through a request's chunks: U = U0 - W S (K split over four lanes), then
// S <- P S + K^T U (the tokens split over two).  W and K of the next chunk are copied meanwhile.  Bound by its two products'
// reads of shared memory and two barriers per chunk.
template <int NC>
struct DcWalkSmem {
    static constexpr int VS = 4 * NC;
    float W[2][HK_C * HK_LD], K[2][HK_C * HK_LD], U[HK_C * VS], S[VS * 144];     // S transposed: [VS][128 + 16]
};

template <int NC>
__global__ void __launch_bounds__(256, 1)
delta_chunk_walk_kernel(const DeltaShape sh, const ChunkScratch cs, float* __restrict__ state, int write_state,
                        const int* __restrict__ positions, const int* __restrict__ q_start, const int* __restrict__ slots, int from) {
    using M = DcWalkSmem<NC>;
    constexpr int VS = M::VS;
    extern __shared__ __align__(16) unsigned char dc_raw[];
    M& m = *reinterpret_cast<M*>(dc_raw);
    ST_PDL_WAIT();
    const int b = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * VS, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int begin = q_start[b], n = q_start[b + 1] - begin, dim = sh.dim, vd = sh.vd;
    if (n < from || positions[begin] < 0) return;
    const int chunks = (n + HK_C - 1) / HK_C;
    const size_t unit0 = (size_t)hk_place(begin, b, from) * sh.H + h;      // and one place, sh.H units, further per chunk
    auto copy = [&](int c) {
        const float* W = cs.W + (unit0 + (size_t)c * sh.H) * HK_C * dim;
        const float* K = cs.K + (unit0 + (size_t)c * sh.H) * HK_C * dim;
        for (int i = tid; i < HK_C * (HK_D / 4); i += 256) {
            const int t = i / (HK_D / 4), e = (i % (HK_D / 4)) * 4;
            if (e < dim) {
                hk_cp16(m.W[c & 1] + t * HK_LD + e, W + t * dim + e);
                hk_cp16(m.K[c & 1] + t * HK_LD + e, K + t * dim + e);
            }
        }
    };
    copy(0);
    asm volatile("cp.async.commit_group;\n" ::);
    // rows of S past dim stay zero, and so do the copied rows' places there
    for (int i = tid; i < VS * 144; i += 256) m.S[i] = 0.f;
    for (int i = tid; i < HK_C * HK_LD; i += 256)
        if (i % HK_LD >= dim) m.W[0][i] = m.W[1][i] = m.K[0][i] = m.K[1][i] = 0.f;
    __syncthreads();
    // for S: a thread's rows 4 ig .., columns NC cg .., tokens of parity kp
    const int kp = lane & 1, cg = (lane >> 1) & 3, ig = warp * 4 + (lane >> 3);
    const bool live = ig * 4 < dim;
    float s[4][NC];
    float* st = state + ((size_t)slots[b] * sh.H + h) * dim * vd + col0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NC; ++j) {
            s[i][j] = live && col0 + cg * NC + j < vd ? __ldcg(st + (size_t)(ig * 4 + i) * vd + cg * NC + j) : 0.f;
            if (kp == 0) m.S[(cg * NC + j) * 144 + ig * 4 + i] = s[i][j];
        }
    // for U: a thread's tokens tr + 16 i, columns NC cu .., dimensions 16 j + 4 kg .. ; of the finished sums it keeps token tr + 16 kg
    const int tr = warp * 2 + (lane & 1), cu = (lane >> 1) & 3, kg = lane >> 3;
    const int t_mine = tr + 16 * kg;
    float u0[NC], p[4];
    auto fetch = [&](int c) {
        const size_t unit = unit0 + (size_t)c * sh.H;
#pragma unroll
        for (int j = 0; j < NC; ++j)
            u0[j] = col0 + cu * NC + j < vd ? __ldcg(cs.U + (unit * HK_C + t_mine) * vd + col0 + cu * NC + j) : 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = live ? __ldcg(cs.P + unit * dim + ig * 4 + i) : 0.f;
    };
    fetch(0);
    for (int c = 0; c < chunks; ++c) {
        const size_t unit = unit0 + (size_t)c * sh.H;
        asm volatile("cp.async.wait_group 0;\n" ::);
        __syncthreads();                                  // W, K of this chunk and S; everyone is done with the chunk before
        if (c + 1 < chunks) copy(c + 1);
        asm volatile("cp.async.commit_group;\n" ::);
        if (kp == 0 && live) {                            // the state before the chunk, for the outputs
            float* dst = cs.S + unit * dim * vd + col0 + cg * NC;
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < NC; ++j)
                    if (col0 + cg * NC + j < vd) dst[(size_t)(ig * 4 + i) * vd + j] = s[i][j];
        }
        float a[4][NC] = {};
        {
            const float* W = m.W[c & 1];
#pragma unroll 2
            for (int e = kg * 4; e < HK_D; e += 16) {
                float4 w[4], x[NC];
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = load4(W + (tr + 16 * i) * HK_LD + e);
#pragma unroll
                for (int j = 0; j < NC; ++j) x[j] = load4(m.S + (cu * NC + j) * 144 + e);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < NC; ++j)
                        a[i][j] += fmaf(w[i].x, x[j].x, fmaf(w[i].y, x[j].y, fmaf(w[i].z, x[j].z, w[i].w * x[j].w)));
            }
        }
#pragma unroll
        for (int j = 0; j < NC; ++j) {
            // four tokens' sums over the four lanes of K: a lane passes on those it does not keep
            const bool up16 = lane & 16, up8 = lane & 8;
            const float x0 = (up16 ? a[2][j] : a[0][j]) + __shfl_xor_sync(0xffffffffu, up16 ? a[0][j] : a[2][j], 16);
            const float x1 = (up16 ? a[3][j] : a[1][j]) + __shfl_xor_sync(0xffffffffu, up16 ? a[1][j] : a[3][j], 16);
            const float y = (up8 ? x1 : x0) + __shfl_xor_sync(0xffffffffu, up8 ? x0 : x1, 8);
            const float u = u0[j] - y;
            m.U[t_mine * VS + cu * NC + j] = u;
            if (col0 + cu * NC + j < vd) cs.U[(unit * HK_C + t_mine) * vd + col0 + cu * NC + j] = u;
        }
        float pc[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) pc[i] = p[i];
        __syncthreads();
        if (c + 1 < chunks) fetch(c + 1);
        float d[4][NC] = {};
        {
            const float* K = m.K[c & 1] + ig * 4;
#pragma unroll 4
            for (int t = kp; t < HK_C; t += 2) {
                const float4 k = load4(K + t * HK_LD);
                float u[NC];
#pragma unroll
                for (int j = 0; j < NC; ++j) u[j] = m.U[t * VS + cg * NC + j];
#pragma unroll
                for (int j = 0; j < NC; ++j) {
                    d[0][j] = fmaf(k.x, u[j], d[0][j]);
                    d[1][j] = fmaf(k.y, u[j], d[1][j]);
                    d[2][j] = fmaf(k.z, u[j], d[2][j]);
                    d[3][j] = fmaf(k.w, u[j], d[3][j]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                d[i][j] += __shfl_xor_sync(0xffffffffu, d[i][j], 1);
                s[i][j] = fmaf(pc[i], s[i][j], d[i][j]);
            }
        if (kp == 0 && live)
#pragma unroll
            for (int j = 0; j < NC; ++j) store4(m.S + (cg * NC + j) * 144 + ig * 4, make_float4(s[0][j], s[1][j], s[2][j], s[3][j]));
    }
    if (write_state && kp == 0 && live)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < NC; ++j)
                if (col0 + cg * NC + j < vd) st[(size_t)(ig * 4 + i) * vd + cg * NC + j] = s[i][j];
    ST_PDL_TRIGGER();
}

// ---- outputs ------------------------------------------------------------------------------------------------------
struct DcOutSmem {
    float Q[HK_C * HK_LD], V[HK_C * HK_LD], A[HK_C * HK_LA], S[2 * HK_SR * HK_LD];
};

__global__ void __launch_bounds__(256, 2)
delta_chunk_out_kernel(const DeltaShape sh, const ChunkScratch cs, float* __restrict__ o, const int* __restrict__ positions,
                       const int* __restrict__ q_start, int n_seqs, int from) {
    extern __shared__ __align__(16) unsigned char dc_raw[];
    DcOutSmem& m = *reinterpret_cast<DcOutSmem*>(dc_raw);
    ST_PDL_WAIT();
    const int place = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int dim = sh.dim, vd = sh.vd;
    int b, first, n;
    if (!hk_find(q_start, positions, n_seqs, from, place, b, first, n)) return;
    const size_t unit = (size_t)place * sh.H + h;
    for (int i = tid; i < HK_C * (HK_D / 4); i += 256) {
        const int t = i / (HK_D / 4), e = (i % (HK_D / 4)) * 4;
        if (e < dim) hk_cp16(m.Q + t * HK_LD + e, cs.Q + (unit * HK_C + t) * dim + e);
        if (e < vd) hk_cp16(m.V + t * HK_LD + e, cs.U + (unit * HK_C + t) * vd + e);
    }
    for (int i = tid; i < HK_C * HK_C / 4; i += 256) {
        const int t = i / (HK_C / 4), e = (i % (HK_C / 4)) * 4;
        hk_cp16(m.A + t * HK_LA + e, cs.A + unit * HK_C * HK_C + 4 * i);
    }
    const float* S0 = cs.S + unit * dim * vd;
    hk_copy_rows(m.S, S0, 0, dim, vd);                     // (its group holds the copies above as well)
    hk_copy_rows(m.S, S0, HK_SR, dim, vd);
    const int row0 = (warp >> 1) * 16 + ((lane & 1) | ((lane >> 4) << 1)), col = (warp & 1) * 64 + ((lane >> 1) & 7) * 4;
    float4 acc[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
    hk_outputs(acc, m.Q, m.A, m.V, m.S, S0, n, dim, vd, row0, col);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int t = row0 + 4 * r;
        if (t >= n) continue;
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (col + 32 * j < vd) store4(o + ((size_t)(first + t) * sh.H + h) * vd + col + 32 * j, acc[r][j]);
    }
    ST_PDL_TRIGGER();
}

long long delta_chunks_floats(int n_tokens, int n_seqs, const DeltaShape& sh) {
    if (sh.dim % 4 || sh.vd % 4 || sh.dim > HK_D || sh.vd > HK_D || sh.H > 65535 || n_seqs > 65535) return 0;
    return hk_places(n_tokens, n_seqs) * sh.H *
           ((long long)HK_C * (3 * sh.dim + sh.vd) + HK_C * HK_C + sh.dim + (long long)sh.dim * sh.vd);
}

int delta_chunks_launch(const float* prep, const DeltaShape& sh, float* scratch, float* state, int write_state, float* o,
                        const int* positions, const int* q_start, const int* slots, int n_tokens, int n_seqs, int from, cudaStream_t s) {
    // (as delta_chunks_floats counts for min(n_seqs, n_tokens / from) requests)
    const long long places = hk_places(n_tokens, hk_longs(n_tokens, n_seqs, from)), units = places * sh.H;
    ChunkScratch cs;
    float* at = scratch;
    auto take = [&](long long per_unit) { float* p = at; at += units * per_unit; return p; };
    cs.W = take((long long)HK_C * sh.dim);
    cs.U = take((long long)HK_C * sh.vd);
    cs.Q = take((long long)HK_C * sh.dim);
    cs.K = take((long long)HK_C * sh.dim);
    cs.A = take(HK_C * HK_C);
    cs.P = take(sh.dim);
    cs.S = take((long long)sh.dim * sh.vd);
    cudaError_t e = cudaFuncSetAttribute(delta_chunk_prepare_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DcPrepareSmem));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_chunk_walk_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DcWalkSmem<2>));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_chunk_walk_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DcWalkSmem<4>));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_chunk_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DcOutSmem));
    if (e != cudaSuccess) return (int)e;
    int rc = st_launch_pdl("delta_chunks", delta_chunk_prepare_kernel, dim3((unsigned)places, sh.H), dim3(256), sizeof(DcPrepareSmem), s,
                           prep, sh, cs, positions, q_start, n_seqs, from);
    if (rc) return rc;
    if ((long long)n_seqs * sh.H * ((sh.vd + 7) / 8) <= st_sm_count())
        rc = st_launch_pdl("delta_chunks", delta_chunk_walk_kernel<2>, dim3((sh.vd + 7) / 8, sh.H, n_seqs), dim3(256),
                           sizeof(DcWalkSmem<2>), s, sh, cs, state, write_state, positions, q_start, slots, from);
    else
        rc = st_launch_pdl("delta_chunks", delta_chunk_walk_kernel<4>, dim3((sh.vd + 15) / 16, sh.H, n_seqs), dim3(256),
                           sizeof(DcWalkSmem<4>), s, sh, cs, state, write_state, positions, q_start, slots, from);
    if (rc) return rc;
    return st_launch_pdl("delta_chunks", delta_chunk_out_kernel, dim3((unsigned)places, sh.H), dim3(256), sizeof(DcOutSmem), s, sh, cs, o,
                         positions, q_start, n_seqs, from);
}
