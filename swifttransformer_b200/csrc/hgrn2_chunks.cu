// The gated linear recurrence of hgrn2.cu over long portions, in chunks of 64 tokens side by side.
//
//   S_t = diag(f_t) S_{t-1} + (1 - f_t) v_t^T,   o_t = S_t^T q_t,   out_t = o_t / sqrt(mean(o_t^2) + eps) * norm_w
//
// Walking the tokens one by one is a chain of a few hundred clocks per token on few blocks (2000 tokens of 16 heads: 1 ms).
// Over a chunk of C tokens after a state S the same is a handful of matrix products:
//
//   S_end = diag(f_1 .. f_C) S + sum_s k~_s v_s^T       k~_s = (1 - f_s) f_{s+1} .. f_C
//   o_t   = S^T (q_t f_1 .. f_t) + sum_{s <= t} A[t][s] v_s,    A[t][s] = sum_i q_t (1 - f_s) f_{s+1} .. f_t
//
// hgrn2_chunk_kv forms every chunk's sum of k~ v^T and its product of gates, hgrn2_chunk_scan walks the chunks (element by
// element: it leaves the state BEFORE a chunk in the chunk's place, and the last state in `state`), hgrn2_chunk_out forms
// the outputs.  Every factor is a product of gates (at most 1), none a quotient, so nothing overflows whatever
// the gates are: A inside 32 tokens is formed with running products, pair by pair; between the two halves of a
// chunk it is a matrix product of q and k~ decayed to the half's border.  All of it is float arithmetic.
//
// Measured on one B200, 2000 tokens of one request, 16 heads of 128 x 128, bfloat16 rows: 155 us (kv 40, scan 18, out 106
// alone) against 1030 for the walk (hgrn2_wide); 1000 tokens of 8 heads 61 / 522; 70 tokens of 16 heads 60 / 52, so portions of
// fewer than about 100 tokens stay with the walk.  kv and out are bound by their instructions
// (two blocks of 256 threads per SM), the scan by its two trips to the second-level cache.  Against 64 bits the states
// are off by 2.9e-7 where the walk's are by 4.0e-7 (fewer roundings in a row).
#include "chunks.cuh"

struct HgrnShape {
    int ld, q_off, f_off, v_off, n_seqs, from, nh, dim, vd;
    float eps;
    const float *f_bias, *lower, *norm_w;
    const int *positions, *q_start, *slots;
};

__device__ __forceinline__ float hk_silu(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float hk_gate(float z, float bias, float lo) { return lo + (1.f - lo) * (1.f / (1.f + expf(-(z + bias)))); }

// ---- a chunk's sum of k~ v^T [dim][vd] and its product of gates [dim] ----------------------------------------
// 256 threads of 8 x 8 sums; lanes l and l ^ 1 share the values they read, l and l ^ 2 the keys (two cycles of shared
// memory per 16-byte read): bound by the multiply-adds.
template <typename T>
__global__ void __launch_bounds__(256, 2)
hgrn2_chunk_kv_kernel(const T* __restrict__ proj, const HgrnShape sh, float* __restrict__ states, float* __restrict__ decays) {
    extern __shared__ __align__(16) float hk_smem[];
    float* K = hk_smem;                                   // [HK_C][HK_LD] gates, then k~
    float* V = K + HK_C * HK_LD;                          // [HK_C][HK_LD]
    ST_PDL_WAIT();
    const int place = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int dim = sh.dim, vd = sh.vd;
    int b, first, n;
    if (!hk_find(sh.q_start, sh.positions, sh.n_seqs, sh.from, place, b, first, n)) return;
    {   // every thread asks for all its pieces before it works on one
        constexpr int N = HK_C * HK_D / 4 / 256;
        const int e = (tid % (HK_D / 4)) * 4, t0 = tid / (HK_D / 4);
        const bool in_f = e < dim, in_v = e < vd;
        const float4 bi = in_f ? load4(sh.f_bias + h * dim + e) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 lo = in_f ? load4(sh.lower + h * dim + e) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 z[N], v[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int t = t0 + i * (256 / (HK_D / 4));
            const T* row = proj + (size_t)(first + min(t, n - 1)) * sh.ld;
            if (in_f) z[i] = load4_cg(row + sh.f_off + h * dim + e);
            if (in_v) v[i] = load4_cg(row + sh.v_off + h * vd + e);
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int t = t0 + i * (256 / (HK_D / 4));
            float4 f = make_float4(1.f, 1.f, 1.f, 1.f);
            if (in_f && t < n)
                f = make_float4(hk_gate(z[i].x, bi.x, lo.x), hk_gate(z[i].y, bi.y, lo.y), hk_gate(z[i].z, bi.z, lo.z), hk_gate(z[i].w, bi.w, lo.w));
            store4(K + t * HK_LD + e, f);
            store4(V + t * HK_LD + e, in_v && t < n ? v[i] : make_float4(0.f, 0.f, 0.f, 0.f));
        }
    }
    __syncthreads();
    {   // two threads per channel, a half of the chunk each: products from the half's end backwards
        const int c = tid & (HK_D - 1), half = tid / HK_D;
        float* at = K + half * HK_H * HK_LD + c;
        float f[HK_H], r = 1.f;
#pragma unroll
        for (int t = 0; t < HK_H; ++t) f[t] = at[t * HK_LD];
        if (!half) {
#pragma unroll
            for (int t = 0; t < HK_H; ++t) r *= K[(HK_H + t) * HK_LD + c];       // the first half decays through the second
        }
        __syncthreads();
#pragma unroll
        for (int t = HK_H - 1; t >= 0; --t) {
            at[t * HK_LD] = (1.f - f[t]) * r;
            r *= f[t];
        }
        if (!half && c < dim) decays[((size_t)place * sh.nh + h) * dim + c] = r;
    }
    __syncthreads();
    const int i0 = (warp >> 1) * 32 + ((lane & 1) | ((lane >> 4) << 1)) * 4, j0 = (warp & 1) * 64 + ((lane >> 1) & 7) * 4;
    if ((warp >> 1) * 32 < dim && (warp & 1) * 64 < vd) {
        float acc[8][8] = {};
#pragma unroll 2
        for (int t = 0; t < n; ++t) {
            const float4 k0 = load4(K + t * HK_LD + i0), k1 = load4(K + t * HK_LD + i0 + 16);
            const float4 v0 = load4(V + t * HK_LD + j0), v1 = load4(V + t * HK_LD + j0 + 32);
            const float k[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
            const float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(k[i], v[j], acc[i][j]);
        }
        float* dst = states + ((size_t)place * sh.nh + h) * dim * vd;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = i0 + (i & 3) + (i >> 2) * 16;
            if (r >= dim) continue;
#pragma unroll
            for (int j = 0; j < 8; j += 4) {
                const int c = j0 + (j >> 2) * 32;
                if (c < vd) store4(dst + (size_t)r * vd + c, make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]));
            }
        }
    }
    ST_PDL_TRIGGER();
}

// ---- the state before every chunk, and the last one ------------------------------------------------------------
__global__ void __launch_bounds__(128)
hgrn2_chunk_scan_kernel(const HgrnShape sh, float* __restrict__ states, const float* __restrict__ decays, float* __restrict__ state) {
    ST_PDL_WAIT();
    const int b = blockIdx.z, h = blockIdx.y, dim = sh.dim, vd = sh.vd;
    const int begin = sh.q_start[b], n = sh.q_start[b + 1] - begin;
    if (n < sh.from || sh.positions[begin] < 0) return;
    const int e = (blockIdx.x * 128 + threadIdx.x) * 4;
    if (e < dim * vd) {
        const int place = hk_place(begin, b, sh.from), chunks = (n + HK_C - 1) / HK_C;
        const size_t step = (size_t)sh.nh * dim * vd, dstep = (size_t)sh.nh * dim;
        float* at = states + (size_t)place * step + (size_t)h * dim * vd + e;
        const float* dec = decays + (size_t)place * dstep + h * dim + e / vd;
        float* st = state + ((size_t)sh.slots[b] * sh.nh + h) * dim * vd + e;
        float4 s = load4_cg(st);
        constexpr int AHEAD = 16;
        for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
            float4 kv[AHEAD];
            float f[AHEAD];
#pragma unroll
            for (int i = 0; i < AHEAD; ++i)
                if (c0 + i < chunks) {
                    kv[i] = load4_cg(at + (size_t)i * step);
                    f[i] = __ldcg(dec + (size_t)i * dstep);
                }
#pragma unroll
            for (int i = 0; i < AHEAD; ++i)
                if (c0 + i < chunks) {
                    store4(at + (size_t)i * step, s);
                    s = make_float4(fmaf(f[i], s.x, kv[i].x), fmaf(f[i], s.y, kv[i].y), fmaf(f[i], s.z, kv[i].z), fmaf(f[i], s.w, kv[i].w));
                }
            at += AHEAD * step;
            dec += AHEAD * dstep;
        }
        store4(st, s);
    }
    ST_PDL_TRIGGER();
}

// ---- outputs ------------------------------------------------------------------------------------------------------
// 256 threads of 4 tokens x 8 values, two blocks per SM (one block's chains of products under the other's sums: with 512
// threads, values of their own memory and one block per SM it took 113 us for 2000 tokens of 16 heads).  The state's
// rows come 16 at a time through two stages of shared memory, asked for before the gates are worked out; the values take the
// place of the gates once those are used up.
struct HkOutSmem {
    float Q[HK_C * HK_LD], F[HK_C * HK_LD], A[HK_C * HK_LA], S[2 * HK_SR * HK_LD], total[HK_D], part[HK_C][2];
};

template <typename T>
__global__ void __launch_bounds__(256, 2)
hgrn2_chunk_out_kernel(const T* __restrict__ proj, const HgrnShape sh, const float* __restrict__ states, T* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char hk_raw[];
    HkOutSmem& m = *reinterpret_cast<HkOutSmem*>(hk_raw);
    ST_PDL_WAIT();
    const int place = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int dim = sh.dim, vd = sh.vd;
    int b, first, n;
    if (!hk_find(sh.q_start, sh.positions, sh.n_seqs, sh.from, place, b, first, n)) return;
    const float* S0 = states + ((size_t)place * sh.nh + h) * dim * vd;
    hk_copy_rows(m.S, S0, 0, dim, vd);
    hk_copy_rows(m.S, S0, HK_SR, dim, vd);
    const int e4 = (tid % (HK_D / 4)) * 4, t4 = tid / (HK_D / 4);         // a thread's pieces: four columns of every eighth row
    constexpr int N = HK_C * HK_D / 4 / 256, TSTEP = 256 / (HK_D / 4);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    {   // every thread asks for all its pieces before it works on one
        const bool in_f = e4 < dim;
        const float4 bi = in_f ? load4(sh.f_bias + h * dim + e4) : zero, lo = in_f ? load4(sh.lower + h * dim + e4) : zero;
        float4 zq[N], z[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const T* row = proj + (size_t)(first + min(t4 + i * TSTEP, n - 1)) * sh.ld;
            if (in_f) { zq[i] = load4_cg(row + sh.q_off + h * dim + e4); z[i] = load4_cg(row + sh.f_off + h * dim + e4); }
        }
        for (int i = tid; i < HK_C * HK_LA / 4; i += 256) store4(m.A + 4 * i, zero);
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int t = t4 + i * TSTEP;
            float4 q = zero, f = make_float4(1.f, 1.f, 1.f, 1.f);
            if (in_f && t < n) {
                q = make_float4(hk_silu(zq[i].x), hk_silu(zq[i].y), hk_silu(zq[i].z), hk_silu(zq[i].w));
                f = make_float4(hk_gate(z[i].x, bi.x, lo.x), hk_gate(z[i].y, bi.y, lo.y), hk_gate(z[i].z, bi.z, lo.z), hk_gate(z[i].w, bi.w, lo.w));
            }
            store4(m.Q + t * HK_LD + e4, q);
            store4(m.F + t * HK_LD + e4, f);
        }
    }
    __syncthreads();
    for (int half = 0; half < HK_C; half += HK_H) {
        if (half >= n) break;
        // A inside a half: a warp takes four s of it, its lanes four channels each; d[k] = (1 - f_s) f_{s+1} .. f_t
        const int s_of[4] = {warp, 15 - warp, 16 + warp, 31 - warp};
        float4 d[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) d[k] = zero;
        const bool up16 = lane & 16, up8 = lane & 8;
        const int mine = up16 ? (up8 ? s_of[3] : s_of[2]) : (up8 ? s_of[1] : s_of[0]);
        const float* qp = m.Q + half * HK_LD + lane * 4;
        const float* fp = m.F + half * HK_LD + lane * 4;
        const int t_end = min(HK_H, n - half);
#pragma unroll 4
        for (int t = 0; t < t_end; ++t) {
            const float4 q = load4(qp + t * HK_LD), f = load4(fp + t * HK_LD);      // (channels past dim: q 0, f 1)
            float o[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (t == s_of[k]) d[k] = make_float4(1.f - f.x, 1.f - f.y, 1.f - f.z, 1.f - f.w);
                else d[k] = make_float4(d[k].x * f.x, d[k].y * f.y, d[k].z * f.z, d[k].w * f.w);
                o[k] = fmaf(q.x, d[k].x, fmaf(q.y, d[k].y, fmaf(q.z, d[k].z, q.w * d[k].w)));
            }
            // four sums over 32 lanes: halves pass on the pair they do not keep, then quarters, then within eight lanes
            const float g0 = __shfl_xor_sync(0xffffffffu, up16 ? o[0] : o[2], 16);
            const float g1 = __shfl_xor_sync(0xffffffffu, up16 ? o[1] : o[3], 16);
            const float x = (up16 ? o[2] : o[0]) + g0, y = (up16 ? o[3] : o[1]) + g1;
            float c = (up8 ? y : x) + __shfl_xor_sync(0xffffffffu, up8 ? x : y, 8);
            c += __shfl_xor_sync(0xffffffffu, c, 4);
            c += __shfl_xor_sync(0xffffffffu, c, 2);
            c += __shfl_xor_sync(0xffffffffu, c, 1);
            if ((lane & 7) == 0 && mine <= t) m.A[(half + t) * HK_LA + half + mine] = c;
        }
    }
    __syncthreads();
    {   // q f_1 .. f_t within each half, and k~ of the first half decayed to its end; all is read before it is overwritten
        const int half = tid / HK_D, c = tid & (HK_D - 1);
        float* fp = m.F + half * HK_H * HK_LD + c;
        float* qp = m.Q + half * HK_H * HK_LD + c;
        float f[HK_H], r = 1.f;
#pragma unroll
        for (int t = 0; t < HK_H; ++t) f[t] = fp[t * HK_LD];
#pragma unroll
        for (int t0 = 0; t0 < HK_H; t0 += 16) {
            float q[16];
#pragma unroll
            for (int t = 0; t < 16; ++t) q[t] = qp[(t0 + t) * HK_LD];
#pragma unroll
            for (int t = 0; t < 16; ++t) {
                r *= f[t0 + t];
                qp[(t0 + t) * HK_LD] = q[t] * r;
            }
        }
        if (!half) {
            m.total[c] = r;
            r = 1.f;
#pragma unroll
            for (int t = HK_H - 1; t >= 0; --t) {
                fp[t * HK_LD] = (1.f - f[t]) * r;
                r *= f[t];
            }
        }
    }
    __syncthreads();
    const int rl = (lane & 1) | ((lane >> 4) << 1), cl = (lane >> 1) & 7;
    if (n > HK_H) {                                       // A between the halves: 2 x 2 sums per thread
        const int t0 = HK_H + (warp >> 1) * 8 + rl, s0 = (warp & 1) * 16 + cl;
        float4 a[2][2];                                   // four chains per sum
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i >> 1][i & 1] = zero;
#pragma unroll 2
        for (int e = 0; e < dim; e += 4) {
            float4 q[2], k[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                q[i] = load4(m.Q + (t0 + 4 * i) * HK_LD + e);
                k[i] = load4(m.F + (s0 + 8 * i) * HK_LD + e);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    a[i][j] = hk_fma4x4(q[i], k[j], a[i][j]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) m.A[(t0 + 4 * i) * HK_LA + s0 + 8 * j] = (a[i][j].x + a[i][j].y) + (a[i][j].z + a[i][j].w);
    }
    __syncthreads();
    {   // the values into the gates' place, and the second half's q from the chunk's start on
        float4 v[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int t = t4 + i * TSTEP;
            v[i] = zero;
            if (e4 < vd && t < n) v[i] = load4_cg(proj + (size_t)(first + t) * sh.ld + sh.v_off + h * vd + e4);
        }
        const float4 w = load4(m.total + e4);
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            float* q = m.Q + (HK_H + t4 + i * TSTEP) * HK_LD + e4;
            const float4 x = load4(q);
            store4(q, make_float4(x.x * w.x, x.y * w.y, x.z * w.z, x.w * w.w));
        }
#pragma unroll
        for (int i = 0; i < N; ++i) store4(m.F + (t4 + i * TSTEP) * HK_LD + e4, v[i]);
    }
    // rows 16 (warp / 2) + rl + 4 i, values 64 (warp % 2) + 4 cl .. and 32 further
    const int row0 = (warp >> 1) * 16 + rl, col = (warp & 1) * 64 + cl * 4;
    float4 acc[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = zero;
    hk_outputs(acc, m.Q, m.A, m.F, m.S, S0, n, dim, vd, row0, col);
    // the norm over a token's values: the eight lanes of a row, then the row's two warps
    const bool has[2] = {col < vd, col + 32 < vd};
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float4 v = acc[r][j];
            if (has[j]) ss += fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, v.w * v.w)));
        }
        ss += __shfl_xor_sync(0xffffffffu, ss, 2);
        ss += __shfl_xor_sync(0xffffffffu, ss, 4);
        ss += __shfl_xor_sync(0xffffffffu, ss, 8);
        if (cl == 0) m.part[row0 + 4 * r][warp & 1] = ss;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int t = row0 + 4 * r;
        if (t >= n) continue;
        const float inv = rsqrtf((m.part[t][0] + m.part[t][1]) / (float)vd + sh.eps);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            if (!has[j]) continue;
            const float4 w = load4(sh.norm_w + col + 32 * j), v = acc[r][j];
            store4(out + ((size_t)(first + t) * sh.nh + h) * vd + col + 32 * j,
                   make_float4(v.x * inv * w.x, v.y * inv * w.y, v.z * inv * w.z, v.w * inv * w.w));
        }
    }
    ST_PDL_TRIGGER();
}

// Floats of scratch for n_seqs requests in chunks in a step of n_tokens tokens, 0: the sizes do not fit (rows of whole 16-byte
// pieces, at most 128 channels and values per head).
ST_EXPORT long long st_hgrn2_chunks_scratch(int n_tokens, int n_seqs, int nh, int dim, int vd) {
    if (n_tokens <= 0 || n_seqs <= 0 || nh <= 0 || dim <= 0 || vd <= 0 || dim % 4 || vd % 4 || dim > HK_D || vd > HK_D) return 0;
    return hk_places(n_tokens, n_seqs) * nh * dim * ((long long)vd + 1);
}

// Arguments as st_hgrn2_scan, for the requests of at least `from` tokens (the others are not touched); scratch: float, 16-byte
// aligned, st_hgrn2_chunks_scratch elements for min(n_seqs, n_tokens / from) requests.  Columns and rows of proj must begin
// on four elements.
ST_EXPORT int st_hgrn2_chunks(const void* proj, int ld, int q_off, int f_off, int v_off, const float* f_bias, const float* lower,
                              const float* norm_w, float eps, float* state, void* out, float* scratch, const int* positions,
                              const int* q_start, const int* slots, int n_tokens, int n_seqs, int from, int nh, int dim, int vd,
                              int dtype, void* stream) {
    if (n_seqs <= 0 || n_tokens <= 0 || n_tokens < from) return 0;
    if (from <= 0) return ST_ERR_BAD_ARG;
    if (st_hgrn2_chunks_scratch(n_tokens, n_seqs, nh, dim, vd) == 0) return ST_ERR_BAD_SIZE;
    if (dtype != 0 && dtype != 1) return ST_ERR_BAD_DTYPE;
    if (ld % 4 || q_off % 4 || f_off % 4 || v_off % 4 || !aligned16(proj) || !aligned16(out) || !aligned16(state) ||
        !aligned16(scratch) || !aligned16(f_bias) || !aligned16(lower) || !aligned16(norm_w)) return ST_ERR_BAD_ARG;
    const long long places = hk_places(n_tokens, hk_longs(n_tokens, n_seqs, from));
    if (nh > 65535 || n_seqs > 65535) return ST_ERR_TOO_LARGE;
    cudaStream_t s = (cudaStream_t)stream;
    HgrnShape sh{ld, q_off, f_off, v_off, n_seqs, from, nh, dim, vd, eps, f_bias, lower, norm_w, positions, q_start, slots};
    float* states = scratch;
    float* decays = scratch + places * nh * dim * vd;
    const size_t kv_smem = sizeof(float) * 2 * HK_C * HK_LD;
#define HK_RUN(T)                                                                                                      \
    do {                                                                                                               \
        cudaError_t e = cudaFuncSetAttribute(hgrn2_chunk_kv_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kv_smem); \
        if (e == cudaSuccess)                                                                                          \
            e = cudaFuncSetAttribute(hgrn2_chunk_out_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(HkOutSmem)); \
        if (e != cudaSuccess) return (int)e;                                                                           \
        int rc = st_launch_pdl("hgrn2_chunks", hgrn2_chunk_kv_kernel<T>, dim3((unsigned)places, nh), dim3(256), kv_smem, s, \
                               (const T*)proj, sh, states, decays);                                                    \
        if (rc) return rc;                                                                                             \
        rc = st_launch_pdl("hgrn2_chunks", hgrn2_chunk_scan_kernel, dim3((dim * vd / 4 + 127) / 128, nh, n_seqs), dim3(128), 0, s, \
                           sh, states, (const float*)decays, state);                                                   \
        if (rc) return rc;                                                                                             \
        return st_launch_pdl("hgrn2_chunks", hgrn2_chunk_out_kernel<T>, dim3((unsigned)places, nh), dim3(256), sizeof(HkOutSmem), s, \
                             (const T*)proj, sh, (const float*)states, (T*)out);                                       \
    } while (0)
    if (dtype == 0) HK_RUN(float);
    HK_RUN(bf16);
#undef HK_RUN
}
