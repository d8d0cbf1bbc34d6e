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
// outputs.  The walk's products run on the tensor cores, every float as the sum of three bfloat16 numbers (float_parts.cuh), the
// rest is float arithmetic, and every factor is a product of decays (at most 1), none a quotient.
//
// Measured on one B200, 2000 tokens of one request, 8 heads of 128 x 128: prepare 53 us, walk 57, out 26, with delta_prepare (20)
// and delta_output (15) 169 us; 16 heads 178 (281 with the walk on the float unit).  The walk on the float unit, 256 threads that
// copied W and K into shared memory, took 110; with the cells' parts formed in the walk itself, 256 threads, 74.  Errors
// against 64 bits: outputs 2.17e-7 (walk on the float unit 2.18e-7, token by token 2.33e-7), states 3.10e-7 (3.11e-7).
// Portions of fewer than 256 tokens stay with the walk token by token.
#include "chunks.cuh"
#include "delta_rule.cuh"
#include "float_parts.cuh"
#include "mma_sync.cuh"

struct ChunkScratch {
    uint4 *W, *K;                          // per (place, head): cells of W and K^T, see below
    float *Q, *A, *P, *S;                  // [64][dim], [64][64], [dim], [dim][vd]
    float* U;                              // [token][head][vd], where the outputs will stand: U0, then U
};

// W [64][dim] and the transpose of K [64][dim] are left operands of the walk's products: cells of 16 x 16, every float as three
// bfloat16 numbers (float_parts.cuh), in the order of mma.m16n8k16's registers: [cell][part][lane] of 16 bytes.  W's cell (token
// block, channel block) is number token * dc_blocks + channel, K^T's (channel block, token block) channel * 4 + token.
#define DC_CELL 96                         // of 16 bytes
__host__ __device__ __forceinline__ int dc_blocks(int dim) { return (dim + 15) / 16; }
__host__ __device__ __forceinline__ long long dc_cells(int dim) { return (long long)dc_blocks(dim) * (HK_C / 16) * DC_CELL; }

// element (t, e) of the unpadded rows of delta_chunk_prepare: pieces of four turned by the row, so that reads of one piece of
// eight rows hit distinct banks
__device__ __forceinline__ int dc_at(int t, int e) { return t * HK_D + (e ^ ((t & 7) << 2)); }

// a lane's part of a cell
__device__ __forceinline__ void dc_cell(uint4* to, float2 a, float2 b, float2 c, float2 d) {
    uint4 hi, mid, lo;
    gf_split(a.x, a.y, hi.x, mid.x, lo.x);
    gf_split(b.x, b.y, hi.y, mid.y, lo.y);
    gf_split(c.x, c.y, hi.z, mid.z, lo.z);
    gf_split(d.x, d.y, hi.w, mid.w, lo.w);
    to[0] = hi;
    to[32] = mid;
    to[64] = lo;
}

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
        float* A = cs.A + unit * HK_C * HK_C;
        if (e4 < dim) {
            const float4 w0 = load4(m.total[0] + e4), w1 = load4(m.total[1] + e4);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int t = t8 + 8 * i;
                float4 q = load4(m.Q + dc_at(t, e4));
                if (i >= 4) q = make_float4(q.x * w0.x, q.y * w0.y, q.z * w0.z, q.w * w0.w);
                store4(Qd + t * dim + e4, q);
            }
            if (t8 == 0) store4(cs.P + unit * dim + e4, make_float4(w0.x * w1.x, w0.y * w1.y, w0.z * w1.z, w0.w * w1.w));
        }
        uint4* K = cs.K + unit * dc_cells(dim);
#pragma unroll 2
        for (int i = warp; i < dc_blocks(dim) * 4; i += 8) {
            const int c = (i >> 2) * 16 + (lane >> 2), t = (i & 3) * 16 + (lane & 3) * 2;
            const float w0 = t < HK_H ? m.total[1][c] : 1.f, w1 = t < HK_H ? m.total[1][c + 8] : 1.f;
            dc_cell(K + i * DC_CELL + lane, make_float2(m.F[dc_at(t, c)] * w0, m.F[dc_at(t + 1, c)] * w0),
                    make_float2(m.F[dc_at(t, c + 8)] * w1, m.F[dc_at(t + 1, c + 8)] * w1), make_float2(m.F[dc_at(t + 8, c)] * w0, m.F[dc_at(t + 9, c)] * w0),
                    make_float2(m.F[dc_at(t + 8, c + 8)] * w1, m.F[dc_at(t + 9, c + 8)] * w1));
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
            float* right = for_w ? m.K : m.F;             // (each x takes the place of its right side)
            const float w0 = for_w ? m.total[0][c] : 1.f;
#pragma unroll 1
            for (int t0 = 0; t0 < HK_C; t0 += 16) {
                float y[16];
#pragma unroll
                for (int t = 0; t < 16; ++t) y[t] = 0.f;
#pragma unroll 2
                for (int s = 0; s < t0; ++s) {
                    const float x = right[dc_at(s, c)];
#pragma unroll
                    for (int t = 0; t < 16; t += 4) {
                        const float4 w = load4(m.AM + s * HK_C + t0 + t);
                        y[t] = fmaf(w.x, x, y[t]);
                        y[t + 1] = fmaf(w.y, x, y[t + 1]);
                        y[t + 2] = fmaf(w.z, x, y[t + 2]);
                        y[t + 3] = fmaf(w.w, x, y[t + 3]);
                    }
                }
                const float wt = t0 >= HK_H ? w0 : 1.f;
                float z[16];
#pragma unroll
                for (int s = 0; s < 16; ++s) z[s] = right[dc_at(t0 + s, c)] * wt;
#pragma unroll
                for (int s = 0; s < 16; ++s) {
                    const float x = m.Q[t0 + s] * (z[s] - y[s]);
                    z[s] = x;
#pragma unroll
                    for (int t = s / 4 * 4; t < 16; t += 4) {
                        if (t + 3 <= s) continue;
                        const float4 w = load4(m.AM + (t0 + s) * HK_C + t0 + t);
                        if (t > s) y[t] = fmaf(w.x, x, y[t]);
                        if (t + 1 > s) y[t + 1] = fmaf(w.y, x, y[t + 1]);
                        if (t + 2 > s) y[t + 2] = fmaf(w.z, x, y[t + 2]);
                        y[t + 3] = fmaf(w.w, x, y[t + 3]);
                    }
                }
#pragma unroll
                for (int s = 0; s < 16; ++s) right[dc_at(t0 + s, c)] = z[s];
            }
        }
    }
    __syncthreads();
    if (e4 < vd)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = t8 + 8 * i;
            if (t < n) store4(cs.U + ((size_t)(first + t) * sh.H + h) * vd + e4, load4(m.F + dc_at(t, e4)));
        }
    uint4* W = cs.W + unit * dc_cells(dim);
    const int blocks = dc_blocks(dim);
#pragma unroll 2
    for (int i = warp; i < blocks * 4; i += 8) {
        const int t = i / blocks * 16 + (lane >> 2), c = i % blocks * 16 + (lane & 3) * 2;
        auto two = [&](int t, int c) { return *reinterpret_cast<const float2*>(m.K + dc_at(t, c)); };
        dc_cell(W + i * DC_CELL + lane, two(t, c), two(t + 8, c), two(t, c + 8), two(t + 8, c + 8));
    }
    ST_PDL_TRIGGER();
}

// ---- the state from chunk to chunk ------------------------------------------------------------------------------
// A block carries 8 NT columns of a head's state through a request's chunks: U = U0 - W S, then S <- P S + K^T U, on the tensor
// cores, every float as three bfloat16 numbers and six products of them per step of sixteen; the highest parts' products have two
// accumulators by turns, the others three, added up in float (one accumulator for all, or one for the highest, is off by more than
// the float unit was).  Eight warps hold W, sixteen tokens and half of the channels each, eight K^T and the state, sixteen channels
// each.  S and U pass between them through shared memory in the order of the right operand's registers, [columns][block of
// 16][part][lane], two barriers per chunk; while eight warps multiply the others ask for the cells of the chunk after next.
//
// Bound by the way of the cells into shared memory (98 KB a chunk and block, some 41 bytes a clock) and by the chain of products,
// sums, parts and barriers.  With the cells in registers straight from memory every load held up the next product: 185 us.
template <int NT>
struct DcWalkSmem {
    uint4 cells[2][16][12][32];            // [chunk & 1][warp][..][lane]: every lane copies what it reads itself
    float2 u0[2][2][NT][128];
    float decay[2][2][256];
    float4 half[4][NT][32];                // W S over the second half of the channels
    uint2 S[NT][8][3][32], U[NT][4][3][32];
};
__device__ __forceinline__ void dc_copy8(float2* dst, const float* src, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(on ? 8 : 0) : "memory");
}
__device__ __forceinline__ void dc_copy4(float* dst, const float* src, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(on ? 4 : 0) : "memory");
}

// the 16 x 8 block x of a right operand, rows (lane >> 2) and + 8, columns 2 (lane & 3) and + 1, as parts in its registers' order
__device__ __forceinline__ void dc_put(uint2 (*dst)[32], const float (&x)[4], int lane) {
    const bool odd = lane & 4;
    uint2 hi, mid, lo;
    const float r0 = __shfl_xor_sync(0xffffffffu, odd ? x[0] : x[1], 4), r1 = __shfl_xor_sync(0xffffffffu, odd ? x[2] : x[3], 4);
    gf_split(odd ? r0 : x[0], odd ? x[1] : r0, hi.x, mid.x, lo.x);
    gf_split(odd ? r1 : x[2], odd ? x[3] : r1, hi.y, mid.y, lo.y);
    const int at = ((lane & 3) * 2 + (lane >> 2 & 1)) * 4 + (lane >> 3);
    dst[0][at] = hi;
    dst[1][at] = mid;
    dst[2][at] = lo;
}
// the six products of a cell with the parts b of a right operand, the highest parts' by turns in one accumulator or the other
__device__ __forceinline__ void dc_products(float (&acc)[6][4], int turn, const uint4 (&a)[3], const uint2 (&b)[3]) {
    mma_bf16(acc[4], &a[1].x, b[1].x, b[1].y);
    mma_bf16(acc[turn & 1], &a[0].x, b[0].x, b[0].y);
    mma_bf16(acc[2], &a[0].x, b[1].x, b[1].y);
    mma_bf16(acc[4], &a[2].x, b[0].x, b[0].y);
    mma_bf16(acc[3], &a[1].x, b[0].x, b[0].y);
    mma_bf16(acc[5], &a[0].x, b[2].x, b[2].y);
}
__device__ __forceinline__ float dc_sum(const float (&acc)[6][4], int i) {
    return ((acc[0][i] + acc[1][i]) + ((acc[2][i] + acc[3][i]) + (acc[4][i] + acc[5][i]))) * GF_DOWN2;
}
// Sums that are not finite, as chains over their n products give them: rows r and r + 8 of the cells from `cells` on, whose columns go
// on by a cell every sixteen, with every `step`-th float from x on and from x + 1 on.  (What is no number stays none.)
__device__ __forceinline__ float dc_chain(const uint4* cells, int r, int n, const float* x, size_t step) {
    float v = 0.f;
    for (int c = 0; c < n && v == v; ++c) {
        const bf16* at = reinterpret_cast<const bf16*>(cells + (c >> 4) * DC_CELL + (r & 7) * 4 + (c >> 1 & 3)) + ((r >> 3) + 2 * (c >> 3 & 1)) * 2 + (c & 1);
        float w = to_f32(at[0]);
        if (fabsf(w) < INFINITY) w = gf_join(w, to_f32(at[256]), to_f32(at[512]));
        v = fmaf(w, __ldcg(x + c * step), v);
    }
    return v;
}

__device__ __noinline__ float4 dc_chains(float4 y, const uint4* cells, int r, int n, const float* x, size_t step) {
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        if (!(fabsf(y.x) < INFINITY)) y.x = dc_chain(cells, r + 8 * (i >> 1), n, x + (i & 1), step);
        y = make_float4(y.y, y.z, y.w, y.x);
    }
    return y;
}

template <int NT>
__global__ void __launch_bounds__(512, 1)
delta_chunk_walk_kernel(const DeltaShape sh, const ChunkScratch cs, float* __restrict__ state, int write_state,
                        const int* __restrict__ positions, const int* __restrict__ q_start, const int* __restrict__ slots, int from) {
    extern __shared__ __align__(16) unsigned char dc_raw[];
    DcWalkSmem<NT>& m = *reinterpret_cast<DcWalkSmem<NT>*>(dc_raw);
    ST_PDL_WAIT();
    const int b = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * 8 * NT, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, w8 = warp & 7;
    const bool second = tid >= 256;                        // K^T and the state; the others W
    const int begin = q_start[b], n = q_start[b + 1] - begin, dim = sh.dim, vd = sh.vd, blocks = dc_blocks(dim);
    if (n < from || positions[begin] < 0) return;
    const int chunks = (n + HK_C - 1) / HK_C, g = lane >> 2, col = col0 + (lane & 3) * 2;
    const size_t unit0 = (size_t)hk_place(begin, b, from) * sh.H + h, cells = dc_cells(dim);      // and sh.H units further per chunk
    // a warp's four cells: of channels 16 w8 and all tokens, or of tokens 16 (w8 % 4) and one half or the other of the channels
    const int tile = w8 & 3, upper = w8 >> 2;
    const int cell0 = second ? w8 * 4 : tile * blocks + 4 * upper, n_cells = second ? (w8 < blocks ? 4 : 0) : min(max(blocks - 4 * upper, 0), 4);
    const uint4* at = (second ? cs.K : cs.W) + unit0 * cells + (size_t)cell0 * DC_CELL;      // those of the chunk at hand
    const size_t u_row = (size_t)sh.H * vd, on = sh.H * cells;
    float* u = cs.U + ((size_t)begin * sh.H + h) * vd;     // the chunk's first row
    float* before = cs.S + unit0 * dim * vd;               // the state before the chunk
    float* st = state + ((size_t)slots[b] * sh.H + h) * dim * vd;
    float s[NT][4];                                        // rows 16 w8 + g and + 8, columns col + 8 i and + 1
    float p[2];                                            // and the rows' decays
    float2 u0[2][NT];                                      // tokens 16 tile + g and + 8, the same columns
    auto copy = [&](int c) {                               // asks for chunk c, in the place of chunk c - 2, had long ago
        asm volatile("" ::: "memory");
        if (c < chunks) {
            const uint4* cell = (second ? cs.K : cs.W) + unit0 * cells + c * on + (size_t)cell0 * DC_CELL + lane;
#pragma unroll 3
            for (int i = 0; i < 3 * n_cells; ++i)
                hk_cp16(reinterpret_cast<float*>(&m.cells[c & 1][warp][i][lane]), reinterpret_cast<const float*>(cell + i * 32));
            if (second) {
                const float* decay = cs.P + (unit0 + (size_t)c * sh.H) * dim;
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int r = 16 * w8 + 8 * x + g;
                    dc_copy4(&m.decay[c & 1][x][tid & 255], decay + (r < dim ? r : 0), r < dim);
                }
            } else if (!upper) {
                const float* row = cs.U + ((size_t)begin * sh.H + h) * vd;
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int i = 0; i < NT; ++i) {
                        const int t = c * HK_C + 16 * tile + g + 8 * r;
                        const bool in = t < n && col + 8 * i < vd;
                        dc_copy8(&m.u0[c & 1][r][i][tid], row + (in ? t * u_row + col + 8 * i : 0), in);
                    }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    auto take = [&](int c) {                               // and has it, in parts
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        if (second) {
#pragma unroll
            for (int x = 0; x < 2; ++x) p[x] = m.decay[c & 1][x][tid & 255];
        } else if (!upper) {
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int i = 0; i < NT; ++i) u0[r][i] = m.u0[c & 1][r][i][tid];
        }
    };
    // the warp's cells times the right operand's blocks from x on
    auto products = [&](int c, const uint2 (*x)[3][32], float (&y)[4]) {
        const uint4* a = m.cells[c & 1][warp][0] + lane;
        float acc[6][4] = {};
#pragma unroll 1
        for (int i = 0; i < n_cells; i += 2) {
            const uint4 f0[3] = {a[0], a[32], a[64]}, f1[3] = {a[96], a[128], a[160]};
            const uint2 v0[3] = {x[i][0][lane], x[i][1][lane], x[i][2][lane]}, v1[3] = {x[i + 1][0][lane], x[i + 1][1][lane], x[i + 1][2][lane]};
            dc_products(acc, 0, f0, v0);
            if (i + 1 < n_cells) dc_products(acc, 1, f1, v1);
            a += 192;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) y[i] = dc_sum(acc, i);
    };
    auto put_state = [&](float* dst) {
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const int c = 16 * w8 + 8 * x + g;
                if (c < dim && col + 8 * i < vd) *reinterpret_cast<float2*>(dst + (size_t)c * vd + col + 8 * i) = make_float2(s[i][2 * x], s[i][2 * x + 1]);
            }
    };
    copy(0);
    if (second) {
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const int c = 16 * w8 + 8 * x + g;
                const bool in = c < dim && col + 8 * i < vd;
                const float2 v = in ? __ldcg(reinterpret_cast<const float2*>(st + (size_t)c * vd + col + 8 * i)) : make_float2(0.f, 0.f);
                s[i][2 * x] = v.x;
                s[i][2 * x + 1] = v.y;
            }
#pragma unroll
        for (int i = 0; i < NT; ++i) dc_put(m.S[i][w8], s[i], lane);
        put_state(before);
    } else {
        copy(1);
        take(0);
    }
    for (int c = 0; c < chunks; ++c) {
        const bool more = c + 1 < chunks;
        __syncthreads();                                   // S
        if (second) {
            copy(c + 1);
            take(c);
        } else {
            float y[NT][4];
#pragma unroll
            for (int j = 0; j < NT; ++j) products(c, &m.S[j][4 * upper], y[j]);
            if (upper) {
#pragma unroll
                for (int j = 0; j < NT; ++j) m.half[tile][j][lane] = make_float4(y[j][0], y[j][1], y[j][2], y[j][3]);
                asm volatile("bar.arrive %0, 64;\n" ::"r"(1 + tile) : "memory");
            } else {
                asm volatile("bar.sync %0, 64;\n" ::"r"(1 + tile) : "memory");
                bool odd = false;
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const float4 z = m.half[tile][j][lane];
                    y[j][0] += z.x; y[j][1] += z.y; y[j][2] += z.z; y[j][3] += z.w;
#pragma unroll
                    for (int x = 0; x < 4; ++x) odd |= !(fabsf(y[j][x]) < INFINITY);
                }
                if (odd)
#pragma unroll
                    for (int j = 0; j < NT; ++j)
                        if (col + 8 * j < vd) {
                            const float4 z = dc_chains(make_float4(y[j][0], y[j][1], y[j][2], y[j][3]), at, g, dim, before + col + 8 * j, vd);
                            y[j][0] = z.x; y[j][1] = z.y; y[j][2] = z.z; y[j][3] = z.w;
                        }
                __syncwarp();
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const float v[4] = {u0[0][j].x - y[j][0], u0[0][j].y - y[j][1], u0[1][j].x - y[j][2], u0[1][j].y - y[j][3]};
                    dc_put(m.U[j][tile], v, lane);
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const int t = 16 * tile + g + 8 * r;
                        if (c * HK_C + t < n && col + 8 * j < vd)
                            *reinterpret_cast<float2*>(u + t * u_row + col + 8 * j) = make_float2(v[2 * r], v[2 * r + 1]);
                    }
                }
            }
        }
        __syncthreads();                                   // U
        if (second) {
            float d[NT][4];
            bool odd = false;
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                products(c, &m.U[i][0], d[i]);
#pragma unroll
                for (int x = 0; x < 4; ++x) odd |= !(fabsf(d[i][x]) < INFINITY);
            }
            if (odd)
#pragma unroll
                for (int i = 0; i < NT; ++i)
                    if (col + 8 * i < vd) {
                        const float4 z = dc_chains(make_float4(d[i][0], d[i][1], d[i][2], d[i][3]), at, g, min(HK_C, n - c * HK_C), u + col + 8 * i, u_row);
                        d[i][0] = z.x; d[i][1] = z.y; d[i][2] = z.z; d[i][3] = z.w;
                    }
            __syncwarp();
            before += (size_t)sh.H * dim * vd;
#pragma unroll
            for (int i = 0; i < NT; ++i) {
#pragma unroll
                for (int x = 0; x < 4; ++x) s[i][x] = fmaf(p[x >> 1], s[i][x], d[i][x]);
                if (more) dc_put(m.S[i][w8], s[i], lane);
            }
            if (more) put_state(before);                   // the state before the next chunk, for the outputs as well
        } else {
            before += (size_t)sh.H * dim * vd;
            if (more) {
                copy(c + 2);
                take(c + 1);
            }
        }
        at += on;
        u += HK_C * u_row;
    }
    if (write_state && second) put_state(st);
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
        if (e < vd && t < n) hk_cp16(m.V + t * HK_LD + e, cs.U + ((size_t)(first + t) * sh.H + h) * vd + e);
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
           (2 * 4 * dc_cells(sh.dim) + (long long)HK_C * sh.dim + HK_C * HK_C + sh.dim + (long long)sh.dim * sh.vd);
}

int delta_chunks_launch(const float* prep, const DeltaShape& sh, float* scratch, float* state, int write_state, float* o,
                        const int* positions, const int* q_start, const int* slots, int n_tokens, int n_seqs, int from, cudaStream_t s) {
    // (as delta_chunks_floats counts for min(n_seqs, n_tokens / from) requests)
    const long long places = hk_places(n_tokens, hk_longs(n_tokens, n_seqs, from)), units = places * sh.H;
    ChunkScratch cs;
    float* at = scratch;
    auto take = [&](long long per_unit) { float* p = at; at += units * per_unit; return p; };
    cs.W = reinterpret_cast<uint4*>(take(4 * dc_cells(sh.dim)));
    cs.K = reinterpret_cast<uint4*>(take(4 * dc_cells(sh.dim)));
    cs.U = o;
    cs.Q = take((long long)HK_C * sh.dim);
    cs.A = take(HK_C * HK_C);
    cs.P = take(sh.dim);
    cs.S = take((long long)sh.dim * sh.vd);
    cudaError_t e = cudaFuncSetAttribute(delta_chunk_prepare_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DcPrepareSmem));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_chunk_walk_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DcWalkSmem<1>));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_chunk_walk_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DcWalkSmem<2>));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_chunk_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DcOutSmem));
    if (e != cudaSuccess) return (int)e;
    int rc = st_launch_pdl("delta_chunks", delta_chunk_prepare_kernel, dim3((unsigned)places, sh.H), dim3(256), sizeof(DcPrepareSmem), s,
                           prep, sh, cs, positions, q_start, n_seqs, from);
    if (rc) return rc;
    if ((long long)n_seqs * sh.H * ((sh.vd + 7) / 8) <= st_sm_count())
        rc = st_launch_pdl("delta_chunks", delta_chunk_walk_kernel<1>, dim3((sh.vd + 7) / 8, sh.H, n_seqs), dim3(512), sizeof(DcWalkSmem<1>), s, sh, cs, state, write_state, positions, q_start, slots, from);
    else
        rc = st_launch_pdl("delta_chunks", delta_chunk_walk_kernel<2>, dim3((sh.vd + 15) / 16, sh.H, n_seqs), dim3(512), sizeof(DcWalkSmem<2>), s, sh, cs, state, write_state, positions, q_start, slots, from);
    if (rc) return rc;
    return st_launch_pdl("delta_chunks", delta_chunk_out_kernel, dim3((unsigned)places, sh.H), dim3(256), sizeof(DcOutSmem), s, sh, cs, o,
                         positions, q_start, n_seqs, from);
}
