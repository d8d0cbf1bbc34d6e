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
// the gates are: A inside 16 tokens is formed with running products, pair by pair; between the blocks of 16 of a
// chunk it is a matrix product of q and k~ decayed to a block's border.
//
// The products run on the tensor cores, every float as the sum of three bfloat16 numbers (float_parts.cuh, gemm_f32.cuh).
//
// Measured on one B200, 2000 tokens of one request, 16 heads of 128 x 128: bfloat16 rows 112 us (kv 28, scan 12, out 70 alone) where
// products on the float unit, divisions one after the other and 35 and 93 KB of code took 158 (kv 42, out 106) and the walk
// (hgrn2_wide) 1030; float rows 142 (160).  333 tokens of 8 heads, 128 x 64: 44 (59); 150 of 16 heads 48 (63).  kv and out are bound
// by their instructions, three or four warps a scheduler (two blocks of 256 threads per SM), the scan by its two trips to the
// second-level cache.  Against 64 bits outputs are off by 1.38e-7 (1.39e-7), states by 2.90e-7 (2.92e-7; the walk's by 4.0e-7).
#include "chunks.cuh"
#include "float_parts.cuh"
#include "mma_sync.cuh"

struct HgrnShape {
    int ld, q_off, f_off, v_off, n_seqs, from, nh, dim, vd;
    float eps;
    const float *f_bias, *lower, *norm_w;
    const int *positions, *q_start, *slots;
};

__device__ __forceinline__ float2 load2_cg(const float* p) { return __ldcg(reinterpret_cast<const float2*>(p)); }
__device__ __forceinline__ float2 load2_cg(const bf16* p) {
    const uint32_t u = __ldcg(reinterpret_cast<const uint32_t*>(p));
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u));
}
__device__ __forceinline__ void store2(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
__device__ __forceinline__ void store2(bf16* p, float a, float b) { *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b); }
__device__ __forceinline__ float hk_gate(float z, float bias, float lo) { return lo + (1.f - lo) * hk_sigmoid(z + bias); }

// ---- the products ------------------------------------------------------------------------------------------------
// Matrices lie in shared memory as bfloat16 planes of their floats' parts (float_parts.cuh: 0 the highest, all times 2^16), rows of HB_LD;
// values that are bfloat16 have one plane, as they are.  A sum of products of two such matrices takes the small products first and is added to what
// it belongs to in float: see gemm_f32.cuh.
#define HB_LD (HK_D + 8)                       // elements: rows 16 bytes apart modulo 128, so that ldmatrix meets no conflict

template <typename T> struct HkValues { static constexpr int PLANES = sizeof(T) == 2 ? 1 : 3; };

// four neighbouring values into the planes at `at`
__device__ __forceinline__ void hk_put(bf16* at, int plane, float4 v, const bf16*) {
    store4(at, v);
}
__device__ __forceinline__ void hk_put(bf16* at, int plane, float4 v, const float*) {
    uint2 h, m, l;
    gf_split(v.x, v.y, h.x, m.x, l.x);
    gf_split(v.z, v.w, h.y, m.y, l.y);
    *reinterpret_cast<uint2*>(at) = h;
    *reinterpret_cast<uint2*>(at + plane) = m;
    *reinterpret_cast<uint2*>(at + 2 * plane) = l;
}
__device__ __forceinline__ float hk_get(const bf16* at, int plane) { return gf_join(to_f32(at[0]), to_f32(at[plane]), to_f32(at[2 * plane])); }

// ---- a chunk's sum of k~ v^T [dim][vd] and its product of gates [dim] ----------------------------------------
// A thread forms k~ of two channels and sixteen tokens: products from its quarter's end backwards, then those of the quarters behind.
// Eight warps of 32 channels x 64 values multiply.  What is not short stands in loops that are not unrolled, with their numbers in
// shared memory: unrolled, the kernel's 260 KB of code took longer to fetch (50 us for 2000 tokens of 16 heads) than to run.
template <typename T>
__global__ void __launch_bounds__(256, 2)
hgrn2_chunk_kv_kernel(const T* __restrict__ proj, const HgrnShape sh, float* __restrict__ states, float* __restrict__ decays) {
    constexpr int PLANES = HkValues<T>::PLANES, PLANE = HK_C * HB_LD;
    extern __shared__ __align__(16) unsigned char hk_kv_raw[];
    bf16* K = reinterpret_cast<bf16*>(hk_kv_raw);         // [3][HK_C][HB_LD]
    bf16* V = K + 3 * PLANE;                              // [PLANES][HK_C][HB_LD]
    float* total = reinterpret_cast<float*>(V + PLANES * PLANE);              // [4][HK_D]
    float* own = total + 4 * HK_D;                        // [HK_C][HK_D] a thread's own tokens: gate logits, then k~
    ST_PDL_WAIT();
    const int place = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int dim = sh.dim, vd = sh.vd;
    int b, first, n;
    if (!hk_find(sh.q_start, sh.positions, sh.n_seqs, sh.from, place, b, first, n)) return;
    const int c = (tid & 63) * 2, quarter = tid >> 6;
    const bool in_f = c < dim;
    own += 16 * quarter * HK_D + c;
    {
        float2 z[16];
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            z[t] = make_float2(0.f, 0.f);
            if (in_f) z[t] = load2_cg(proj + (size_t)(first + min(16 * quarter + t, n - 1)) * sh.ld + sh.f_off + h * dim + c);
        }
        constexpr int N = HK_C * HK_D / 4 / 256;
        const int e = (tid % (HK_D / 4)) * 4, t0 = tid / (HK_D / 4);
        float4 v[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int t = t0 + i * (256 / (HK_D / 4));
            v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (e < vd && t < n) v[i] = load4_cg(proj + (size_t)(first + t) * sh.ld + sh.v_off + h * vd + e);
        }
#pragma unroll
        for (int t = 0; t < 16; ++t) *reinterpret_cast<float2*>(own + t * HK_D) = z[t];
#pragma unroll
        for (int i = 0; i < N; ++i) hk_put(V + (t0 + i * (256 / (HK_D / 4))) * HB_LD + e, PLANE, v[i], (const T*)nullptr);
    }
    {
        const float b0 = in_f ? sh.f_bias[h * dim + c] : 0.f, b1 = in_f ? sh.f_bias[h * dim + c + 1] : 0.f;
        const float l0 = in_f ? sh.lower[h * dim + c] : 0.f, l1 = in_f ? sh.lower[h * dim + c + 1] : 0.f;
        float r0 = 1.f, r1 = 1.f;
#pragma unroll 2
        for (int t = 15; t >= 0; --t) {
            const bool on = in_f && 16 * quarter + t < n;
            const float2 z = *reinterpret_cast<const float2*>(own + t * HK_D);
            const float f0 = on ? hk_gate(z.x, b0, l0) : 1.f, f1 = on ? hk_gate(z.y, b1, l1) : 1.f;
            *reinterpret_cast<float2*>(own + t * HK_D) = make_float2((1.f - f0) * r0, (1.f - f1) * r1);
            r0 *= f0;
            r1 *= f1;
        }
        total[quarter * HK_D + c] = r0;
        total[quarter * HK_D + c + 1] = r1;
    }
    __syncthreads();
    {
        float r0 = 1.f, r1 = 1.f;
        for (int q = quarter + 1; q < 4; ++q) { r0 *= total[q * HK_D + c]; r1 *= total[q * HK_D + c + 1]; }
#pragma unroll 4
        for (int t = 0; t < 16; ++t) {
            const float2 k = *reinterpret_cast<const float2*>(own + t * HK_D);
            uint32_t hi, mid, lo;
            gf_split(k.x * r0, k.y * r1, hi, mid, lo);
            uint32_t* at = reinterpret_cast<uint32_t*>(K + (16 * quarter + t) * HB_LD + c);
            at[0] = hi;
            at[PLANE / 2] = mid;
            at[PLANE] = lo;
        }
        if (quarter == 0 && c < dim) {
            float* at = decays + ((size_t)place * sh.nh + h) * dim + c;
            at[0] = total[c] * r0;
            at[1] = total[c + 1] * r1;
        }
    }
    __syncthreads();
    const int m0 = (warp >> 1) * 32, n0 = (warp & 1) * 64;
    if (m0 < dim && n0 < vd) {
        float acc[2][8][4] = {};
        constexpr int N_PROD = PLANES == 1 ? 3 : 6;
        constexpr int KP[6] = {2, PLANES == 1 ? 1 : 0, PLANES == 1 ? 0 : 1, 1, 0, 0}, VP[6] = {0, PLANES == 1 ? 0 : 2, PLANES == 1 ? 0 : 1, 0, 1, 0};
#pragma unroll
        for (int x = 0; x < N_PROD; ++x)
            for (int t = 0; t < n; t += 16) {
                uint32_t a[2][4];
                const bf16* ka = K + KP[x] * PLANE + (t + (lane & 7) + ((lane >> 4) << 3)) * HB_LD + m0 + ((lane >> 3) & 1) * 8;
#pragma unroll
                for (int mt = 0; mt < 2; ++mt) ldmatrix_x4_trans(a[mt][0], a[mt][1], a[mt][2], a[mt][3], ka + 16 * mt);
                const bf16* va = V + VP[x] * PLANE + (t + (lane & 15)) * HB_LD + n0 + (lane >> 4) * 8;
#pragma unroll
                for (int nt = 0; nt < 4; ++nt) {
                    uint32_t b0, b1, b2, b3;
                    ldmatrix_x4_trans(b0, b1, b2, b3, va + 16 * nt);
#pragma unroll
                    for (int mt = 0; mt < 2; ++mt) {
                        mma_bf16(acc[mt][2 * nt], a[mt], b0, b1);
                        mma_bf16(acc[mt][2 * nt + 1], a[mt], b2, b3);
                    }
                }
            }
        const int g = lane >> 2, t2 = (lane & 3) * 2;
        float* dst = states + ((size_t)place * sh.nh + h) * dim * vd;
        bool odd = false;
#pragma unroll
        for (int x = 0; x < 32; ++x) {
            const int mt = x >> 4, nt = x >> 1 & 7, half = x & 1;
            const int r = m0 + 16 * mt + 8 * half + g, col = n0 + 8 * nt + t2;
            const float down = PLANES == 1 ? GF_DOWN : GF_DOWN2;
            const float2 v = make_float2(acc[mt][nt][2 * half] * down, acc[mt][nt][2 * half + 1] * down);
            odd |= !(fabsf(v.x) < INFINITY && fabsf(v.y) < INFINITY);
            if (r < dim && col < vd) *reinterpret_cast<float2*>(dst + (size_t)r * vd + col) = v;
        }
        // Sums that are not finite: what a chain over the tokens gives.  It takes the values from the rows: the parts of an infinite
        // one, or of a float beyond the largest bfloat16, do not add up to it.  (k~ is at most 1 where gates are.)
        if (odd)
#pragma unroll 1
            for (int x = 0; x < 64; ++x) {
                const int r = m0 + 16 * (x >> 5) + 8 * (x >> 1 & 1) + g, col = n0 + 8 * (x >> 2 & 7) + t2 + (x & 1);
                if (r >= dim || col >= vd || fabsf(dst[(size_t)r * vd + col]) < INFINITY) continue;
                const T* value = proj + (size_t)first * sh.ld + sh.v_off + h * vd + col;
                float v = 0.f;
#pragma unroll 1
                for (int t = 0; t < n; ++t) v = fmaf(hk_get(K + t * HB_LD + r, PLANE), load1_cg(value + (size_t)t * sh.ld), v);
                dst[(size_t)r * vd + col] = v;
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
// A chunk in four blocks of sixteen tokens.  A inside a block is formed with running products, pair by pair: a warp takes two s of
// it, s and 15 - s, so that all warps walk over seventeen t, sixteen lanes eight channels each.  Between blocks it is a matrix
// product of q decayed from its block's start and k~ decayed to its block's end and on to the other's start.  Then eight warps of
// sixteen tokens x 64 values multiply q, decayed from the chunk's start, with the state, whose rows come sixteen at a time through two
// stages of planes, and A with the values.  Rows and results that are floats take multiply-adds for these two products
// instead (hk_outputs): with three planes of values one block fits an SM (157 us against 142).  Loops are unrolled only where registers demand it: see hgrn2_chunk_kv_kernel.
struct HkOutSmem {
    float Q[HK_C * HK_LD], F[HK_C * HK_LD], A[HK_C * HK_LA];
    bf16 S[2][3][16 * HB_LD];                             // (and the partial sums of A between blocks, [4][12][128])
    float total[4][HK_D], part[HK_C][2];
};                                                        // (the values take the gates' place)
static_assert(sizeof(HkOutSmem) <= 113 * 1024, "two blocks per SM");
static_assert(4 * 12 * 128 * 4 <= 2 * 3 * 16 * HB_LD * 2 && 256 * 16 * 4 <= 2 * 3 * 16 * HB_LD * 2, "the partial sums fit, and sixteen sums a thread");

// what an output is made of where its sum is not finite: q of its row from the chunk's start, the state, A of its row, the values and
// their parts
template <typename T>
struct HkOdd {
    const float *q, *state, *a;
    const bf16* values;
    const T* rows;
    int dim, vd, ld, odd;
};
template <typename T>
__device__ __noinline__ float hk_odd_output(const HkOdd<T>& o, float x, int t, int col) {
    if (!(fabsf(x) < INFINITY)) {                         // chains over the channels and over the tokens up to the row
        x = 0.f;
        for (int c = 0; c < o.dim; ++c) x = fmaf(o.q[t * HK_LD + c], __ldcg(o.state + (size_t)c * o.vd + col), x);
        for (int s = 0; s <= t; ++s) x = fmaf(o.a[t * HK_LA + s], to_f32(o.values[s * HB_LD + col]), x);
    }
    if (o.odd)                                            // the values that stayed out of the products
        for (int s = 0; s <= t; ++s) {
            const float v = to_f32(o.rows[(size_t)s * o.ld + col]);
            if (!(fabsf(v) < INFINITY)) x = fmaf(o.a[t * HK_LA + s], v, x);
        }
    return x;
}
// an element of A between blocks i and j where its sum is not finite
__device__ __noinline__ inline float hk_odd_between(const float* q, const float* k, const float* f1, const float* f2, int dim, bool one, bool two) {
    float a = 0.f;
    for (int c = 0; c < dim; ++c) {
        float x = k[c];
        if (one) x *= f1[c];
        if (two) x *= f2[c];
        a = fmaf(q[c], x, a);
    }
    return a;
}

template <typename T>
__global__ void __launch_bounds__(256, 2)
hgrn2_chunk_out_kernel(const T* __restrict__ proj, const HgrnShape sh, const float* __restrict__ states, T* __restrict__ out) {
    constexpr bool FLOATS = sizeof(T) == 4;
    constexpr int S_PLANE = 16 * HB_LD;
    extern __shared__ __align__(16) unsigned char hk_raw[];
    HkOutSmem& m = *reinterpret_cast<HkOutSmem*>(hk_raw);
    bf16* V = reinterpret_cast<bf16*>(m.F);
    ST_PDL_WAIT();
    const int place = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t2 = (lane & 3) * 2;
    const int dim = sh.dim, vd = sh.vd;
    int b, first, n;
    if (!hk_find(sh.q_start, sh.positions, sh.n_seqs, sh.from, place, b, first, n)) return;
    const float* S0 = states + ((size_t)place * sh.nh + h) * dim * vd;
    const int e4 = (tid % (HK_D / 4)) * 4, t4 = tid / (HK_D / 4);         // a thread's pieces: four columns of every eighth row
    constexpr int N = HK_C * HK_D / 4 / 256, TSTEP = 256 / (HK_D / 4);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    // the state's rows 16 i .. 16 i + 15: a thread has eight columns of one, asked for one step ahead of their parts
    const int sr = tid >> 4, sc = (tid & 15) * 8;
    float4 s_next[2];
    auto ask = [&](int i) {
        const int r = 16 * i + sr;
#pragma unroll
        for (int j = 0; j < 2; ++j) s_next[j] = r < dim && sc + 4 * j < vd ? load4_cg(S0 + (size_t)r * vd + sc + 4 * j) : zero;
    };
    auto put = [&](int i) {
        uint4 hi, mid, lo;
        gf_split(s_next[0].x, s_next[0].y, hi.x, mid.x, lo.x);
        gf_split(s_next[0].z, s_next[0].w, hi.y, mid.y, lo.y);
        gf_split(s_next[1].x, s_next[1].y, hi.z, mid.z, lo.z);
        gf_split(s_next[1].z, s_next[1].w, hi.w, mid.w, lo.w);
        bf16* at = m.S[i & 1][0] + sr * HB_LD + sc;
        *reinterpret_cast<uint4*>(at) = hi;
        *reinterpret_cast<uint4*>(at + S_PLANE) = mid;
        *reinterpret_cast<uint4*>(at + 2 * S_PLANE) = lo;
    };
    {   // every thread asks for all its pieces before it works on one
        const bool in_f = e4 < dim;
        const float4 bi = in_f ? load4(sh.f_bias + h * dim + e4) : zero, lo = in_f ? load4(sh.lower + h * dim + e4) : zero;
        float4 zq[N], z[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const T* row = proj + (size_t)(first + min(t4 + i * TSTEP, n - 1)) * sh.ld;
            zq[i] = z[i] = zero;
            if (in_f) { zq[i] = load4_cg(row + sh.q_off + h * dim + e4); z[i] = load4_cg(row + sh.f_off + h * dim + e4); }
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            store4(m.Q + (t4 + i * TSTEP) * HK_LD + e4, zq[i]);
            store4(m.F + (t4 + i * TSTEP) * HK_LD + e4, z[i]);
        }
#pragma unroll 1
        for (int t = t4; t < HK_C; t += TSTEP) {
            float4 q = load4(m.Q + t * HK_LD + e4), f = load4(m.F + t * HK_LD + e4);
            const bool on = in_f && t < n;
            q = on ? make_float4(hk_silu(q.x), hk_silu(q.y), hk_silu(q.z), hk_silu(q.w)) : zero;
            f = on ? make_float4(hk_gate(f.x, bi.x, lo.x), hk_gate(f.y, bi.y, lo.y), hk_gate(f.z, bi.z, lo.z), hk_gate(f.w, bi.w, lo.w))
                   : make_float4(1.f, 1.f, 1.f, 1.f);
            store4(m.Q + t * HK_LD + e4, q);
            store4(m.F + t * HK_LD + e4, f);
        }
    }
    if (!FLOATS) ask(0);
    __syncthreads();
    // A inside a block of sixteen: half a warp has every second block; channels 4 o .. and 64 + 4 o .. of lane o
#pragma unroll 1
    for (int blk = lane >> 4; blk < 4; blk += 2) {
        const float* qp = m.Q + blk * 16 * HK_LD + (lane & 15) * 4;
        const float* fp = m.F + blk * 16 * HK_LD + (lane & 15) * 4;
#pragma unroll 1
        for (int x = 0; x < 2; ++x) {
            const int s = x ? 15 - warp : warp;
            float4 d0 = zero, d1 = zero;                  // (1 - f_s) f_{s+1} .. f_t
            float o[16];
#pragma unroll
            for (int t = 0; t < 16; ++t) {
                o[t] = 0.f;
                if (t < s) continue;                      // (the same for the whole warp)
                const float4 f0 = load4(fp + t * HK_LD), f1 = load4(fp + t * HK_LD + 64);
                const float4 q0 = load4(qp + t * HK_LD), q1 = load4(qp + t * HK_LD + 64);
                if (t == s) {
                    d0 = make_float4(1.f - f0.x, 1.f - f0.y, 1.f - f0.z, 1.f - f0.w);
                    d1 = make_float4(1.f - f1.x, 1.f - f1.y, 1.f - f1.z, 1.f - f1.w);
                } else {
                    d0 = make_float4(d0.x * f0.x, d0.y * f0.y, d0.z * f0.z, d0.w * f0.w);
                    d1 = make_float4(d1.x * f1.x, d1.y * f1.y, d1.z * f1.z, d1.w * f1.w);
                }
                o[t] = fmaf(q0.x, d0.x, fmaf(q0.y, d0.y, fmaf(q0.z, d0.z, q0.w * d0.w))) +
                       fmaf(q1.x, d1.x, fmaf(q1.y, d1.y, fmaf(q1.z, d1.z, q1.w * d1.w)));
            }
            // sixteen sums over sixteen lanes: halves pass on the eight they do not keep, then four, two, one
            float y[8], z[4], u[2];
            const bool up8 = lane & 8, up4 = lane & 4, up2 = lane & 2, up1 = lane & 1;
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = (up8 ? o[8 + i] : o[i]) + __shfl_xor_sync(0xffffffffu, up8 ? o[i] : o[8 + i], 8);
#pragma unroll
            for (int i = 0; i < 4; ++i) z[i] = (up4 ? y[4 + i] : y[i]) + __shfl_xor_sync(0xffffffffu, up4 ? y[i] : y[4 + i], 4);
#pragma unroll
            for (int i = 0; i < 2; ++i) u[i] = (up2 ? z[2 + i] : z[i]) + __shfl_xor_sync(0xffffffffu, up2 ? z[i] : z[2 + i], 2);
            const float a = (up1 ? u[1] : u[0]) + __shfl_xor_sync(0xffffffffu, up1 ? u[0] : u[1], 1);
            const int t = lane & 15;
            m.A[(blk * 16 + t) * HK_LA + blk * 16 + s] = t < s ? 0.f : a;
        }
    }
    __syncthreads();
    {   // q f_1 .. f_t and k~ to the end within each block; all of a block is read before it is overwritten
        const int c = tid & (HK_D - 1);
#pragma unroll 1
        for (int j = 0; j < 2; ++j) {
            const int blk = (tid / HK_D) * 2 + j;
            float* fp = m.F + blk * 16 * HK_LD + c;
            float* qp = m.Q + blk * 16 * HK_LD + c;
            float f[16], q[16], r = 1.f;
#pragma unroll
            for (int t = 0; t < 16; ++t) { f[t] = fp[t * HK_LD]; q[t] = qp[t * HK_LD]; }
#pragma unroll
            for (int t = 0; t < 16; ++t) { r *= f[t]; qp[t * HK_LD] = q[t] * r; }
            m.total[blk][c] = r;
            r = 1.f;
#pragma unroll
            for (int t = 15; t >= 0; --t) { fp[t * HK_LD] = (1.f - f[t]) * r; r *= f[t]; }
        }
    }
    __syncthreads();
    float* partial = reinterpret_cast<float*>(m.S);
    constexpr int BI[6] = {1, 2, 2, 3, 3, 3}, BJ[6] = {0, 0, 1, 0, 1, 2};
    if (n > 16) {                                         // A between the blocks: a warp has 32 channels and eight s of every block
        const int c0 = (warp >> 1) * 32, sb = (warp & 1) * 8;
        float acc[6][4] = {};
#pragma unroll 1
        for (int c = c0; c < min(c0 + 32, dim); c += 16) {
            float2 kd[3][2];
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
                for (int x = 0; x < 2; ++x) kd[j][x] = *reinterpret_cast<const float2*>(m.F + (16 * j + sb + g) * HK_LD + c + 8 * x + t2);
            float2 f1[2], f2[2];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                f1[x] = *reinterpret_cast<const float2*>(m.total[1] + c + 8 * x + t2);
                f2[x] = *reinterpret_cast<const float2*>(m.total[2] + c + 8 * x + t2);
            }
#pragma unroll
            for (int i = 1; i < 4; ++i) {
                if (16 * i >= n) break;
                uint32_t qh[4], qm[4], ql[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float2 q = *reinterpret_cast<const float2*>(m.Q + (16 * i + 8 * (r & 1) + g) * HK_LD + c + 8 * (r >> 1) + t2);
                    gf_split(q.x, q.y, qh[r], qm[r], ql[r]);
                }
#pragma unroll
                for (int j = 0; j < i; ++j) {
                    uint32_t kh[2], km[2], kl[2];
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        float2 k = kd[j][x];
                        if (j == 0 && i >= 2) { k.x *= f1[x].x; k.y *= f1[x].y; }
                        if (j <= 1 && i == 3) { k.x *= f2[x].x; k.y *= f2[x].y; }
                        gf_split(k.x, k.y, kh[x], km[x], kl[x]);
                    }
                    float a[4] = {0.f, 0.f, 0.f, 0.f};
                    mma_bf16(a, ql, kh[0], kh[1]);
                    mma_bf16(a, qh, kl[0], kl[1]);
                    mma_bf16(a, qm, km[0], km[1]);
                    mma_bf16(a, qm, kh[0], kh[1]);
                    mma_bf16(a, qh, km[0], km[1]);
                    mma_bf16(a, qh, kh[0], kh[1]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[i * (i - 1) / 2 + j][e] = fmaf(a[e], GF_DOWN2, acc[i * (i - 1) / 2 + j][e]);
                }
            }
        }
#pragma unroll
        for (int x = 0; x < 6; ++x) {
            float* dst = partial + ((warp >> 1) * 12 + 2 * x + (warp & 1)) * 128 + g * 8 + t2;
            *reinterpret_cast<float2*>(dst) = make_float2(acc[x][0], acc[x][1]);
            *reinterpret_cast<float2*>(dst + 64) = make_float2(acc[x][2], acc[x][3]);
        }
    }
    __syncthreads();
    if (n > 16)
#pragma unroll
        for (int x = 0; x < 6; ++x) {
            const int e = tid, t = 16 * BI[x] + ((e >> 3) & 15), s = 16 * BJ[x] + (e >> 7) * 8 + (e & 7);
            const float* src = partial + (2 * x + (e >> 7)) * 128 + (e & 127);
            float a = ((src[0] + src[12 * 128]) + src[24 * 128]) + src[36 * 128];
            if (!(fabsf(a) < INFINITY))
                a = hk_odd_between(m.Q + t * HK_LD, m.F + s * HK_LD, m.total[1], m.total[2], dim, BJ[x] == 0 && BI[x] >= 2, BJ[x] <= 1 && BI[x] == 3);
            m.A[t * HK_LA + s] = a;
        }
    __syncthreads();
    // Values that are not finite stay out of the products, where a token's would reach the rows before it (zero times such a
    // number is none), and are added to the rows behind them one by one.
    bool odd = false;
    {   // the values' planes, and q from the chunk's start on
        float4 v[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int t = t4 + i * TSTEP;
            v[i] = zero;
            if (e4 < vd && t < n) v[i] = load4_cg(proj + (size_t)(first + t) * sh.ld + sh.v_off + h * vd + e4);
        }
        const float4 w0 = load4(m.total[0] + e4), w1 = load4(m.total[1] + e4), w2 = load4(m.total[2] + e4);
        float4 w = w0;
#pragma unroll
        for (int i = 2; i < N; ++i) {                     // rows 8 i + t4: block i / 2
            if (i == 4) w = make_float4(w.x * w1.x, w.y * w1.y, w.z * w1.z, w.w * w1.w);
            if (i == 6) w = make_float4(w.x * w2.x, w.y * w2.y, w.z * w2.z, w.w * w2.w);
            float* q = m.Q + (t4 + i * TSTEP) * HK_LD + e4;
            const float4 x = load4(q);
            store4(q, make_float4(x.x * w.x, x.y * w.y, x.z * w.z, x.w * w.w));
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            if (FLOATS) {
                store4(m.F + (t4 + i * TSTEP) * HK_LD + e4, v[i]);
                continue;
            }
            if (!(fabsf(v[i].x) < INFINITY)) { v[i].x = 0.f; odd = true; }
            if (!(fabsf(v[i].y) < INFINITY)) { v[i].y = 0.f; odd = true; }
            if (!(fabsf(v[i].z) < INFINITY)) { v[i].z = 0.f; odd = true; }
            if (!(fabsf(v[i].w) < INFINITY)) { v[i].w = 0.f; odd = true; }
            store4(V + (t4 + i * TSTEP) * HB_LD + e4, v[i]);
        }
    }
    if constexpr (FLOATS) {
        float* ring = reinterpret_cast<float*>(m.S);
        hk_copy_rows(ring, S0, 0, dim, vd);
        hk_copy_rows(ring, S0, HK_SR, dim, vd);
        // rows 16 (warp / 2) + rl + 4 i, values 64 (warp % 2) + 4 cl .. and 32 further
        const int rl = (lane & 1) | ((lane >> 4) << 1), cl = (lane >> 1) & 7, row0 = (warp >> 1) * 16 + rl, col = (warp & 1) * 64 + cl * 4;
        float4 acc[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = zero;
        hk_outputs(acc, m.Q, m.A, m.F, ring, S0, n, dim, vd, row0, col);
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
            const float inv = hk_rsqrt((m.part[t][0] + m.part[t][1]) / (float)vd + sh.eps);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (!has[j]) continue;
                const float4 w = load4(sh.norm_w + col + 32 * j), v = acc[r][j];
                store4(out + ((size_t)(first + t) * sh.nh + h) * vd + col + 32 * j,
                       make_float4(v.x * inv * w.x, v.y * inv * w.y, v.z * inv * w.z, v.w * inv * w.w));
            }
        }
        ST_PDL_TRIGGER();
        return;
    }
    put(0);
    ask(1);
    odd = __syncthreads_or(odd);
    const int row0 = (warp >> 1) * 16, n0 = (warp & 1) * 64;
    const bool active = row0 < n && n0 < vd;
    float acc[8][4] = {};
    auto parts_of = [&](const float* at, int ld, uint32_t* hi, uint32_t* mid, uint32_t* lo) {       // an A fragment from floats
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float2 x = *reinterpret_cast<const float2*>(at + (8 * (r & 1) + g) * ld + 8 * (r >> 1) + t2);
            gf_split(x.x, x.y, hi[r], mid[r], lo[r]);
        }
    };
#pragma unroll 1
    for (int i = 0; 16 * i < dim; ++i) {
        __syncthreads();                                  // stage i is written, and everyone is done with the one before
        if (16 * (i + 1) < dim) {
            put(i + 1);
            ask(i + 2);
        }
        if (!active) continue;
        uint32_t xh[4], xm[4], xl[4];
        parts_of(m.Q + row0 * HK_LD + 16 * i, HK_LD, xh, xm, xl);
        const bf16* sa = m.S[i & 1][0] + (lane & 15) * HB_LD + n0 + (lane >> 4) * 8;
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            uint32_t sh_[4], sm[4], sl[4];
            ldmatrix_x4_trans(sh_[0], sh_[1], sh_[2], sh_[3], sa + 16 * nt);
            ldmatrix_x4_trans(sm[0], sm[1], sm[2], sm[3], sa + 16 * nt + S_PLANE);
            ldmatrix_x4_trans(sl[0], sl[1], sl[2], sl[3], sa + 16 * nt + 2 * S_PLANE);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float c[4] = {0.f, 0.f, 0.f, 0.f};
                mma_bf16(c, xl, sh_[2 * j], sh_[2 * j + 1]);
                mma_bf16(c, xh, sl[2 * j], sl[2 * j + 1]);
                mma_bf16(c, xm, sm[2 * j], sm[2 * j + 1]);
                mma_bf16(c, xm, sh_[2 * j], sh_[2 * j + 1]);
                mma_bf16(c, xh, sm[2 * j], sm[2 * j + 1]);
                mma_bf16(c, xh, sh_[2 * j], sh_[2 * j + 1]);
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[2 * nt + j][e] = fmaf(c[e], GF_DOWN2, acc[2 * nt + j][e]);
            }
        }
    }
    if (active)
#pragma unroll 1
        for (int s = 0; s <= row0; s += 16) {             // (A is zero above its diagonal)
            uint32_t ah[4], am[4], al[4];
            parts_of(m.A + row0 * HK_LA + s, HK_LA, ah, am, al);
            const bf16* va = V + (s + (lane & 15)) * HB_LD + n0 + (lane >> 4) * 8;
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                uint32_t v[4];
                ldmatrix_x4_trans(v[0], v[1], v[2], v[3], va + 16 * nt);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    float c[4] = {0.f, 0.f, 0.f, 0.f};
                    mma_bf16(c, al, v[2 * j], v[2 * j + 1]);
                    mma_bf16(c, am, v[2 * j], v[2 * j + 1]);
                    mma_bf16(c, ah, v[2 * j], v[2 * j + 1]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[2 * nt + j][e] = fmaf(c[e], GF_DOWN, acc[2 * nt + j][e]);
                }
            }
        }
    {   // sums that are not finite give way (sixteen at a time by way of the state's place, so that there is one piece of code for it)
        bool any = odd;
#pragma unroll
        for (int x = 0; x < 32; ++x) any |= !(fabsf(acc[x >> 2][x & 3]) < INFINITY);
        if (__syncthreads_or(any)) {
            const HkOdd<T> what = {m.Q, S0, m.A, V, proj + (size_t)first * sh.ld + sh.v_off + h * vd, dim, vd, sh.ld, odd};
            float* own = partial + tid;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
#pragma unroll
                for (int x = 0; x < 16; ++x) own[256 * x] = acc[4 * half + (x >> 2)][x & 3];
#pragma unroll 1
                for (int x = 0; x < 16; ++x) {
                    const int t = row0 + 8 * (x >> 1 & 1) + g, col = n0 + 8 * (4 * half + (x >> 2)) + t2 + (x & 1);
                    if (active && col < vd && t < n) own[256 * x] = hk_odd_output<T>(what, own[256 * x], t, col);
                }
#pragma unroll
                for (int x = 0; x < 16; ++x) acc[4 * half + (x >> 2)][x & 3] = own[256 * x];
            }
        }
    }
    // the norm over a token's values: four lanes, two warps
    float ss[2] = {0.f, 0.f};
    if (active) {
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (n0 + 8 * nt + t2 < vd) ss[e >> 1] = fmaf(acc[nt][e], acc[nt][e], ss[e >> 1]);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        ss[r] += __shfl_xor_sync(0xffffffffu, ss[r], 1);
        ss[r] += __shfl_xor_sync(0xffffffffu, ss[r], 2);
        if ((lane & 3) == 0) m.part[row0 + 8 * r + g][warp & 1] = ss[r];
    }
    __syncthreads();
    const float by_vd = 1.f / (float)vd;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int t = row0 + 8 * r + g;
        if (!active || t >= n) continue;
        const float inv = hk_rsqrt((m.part[t][0] + m.part[t][1]) * by_vd + sh.eps);
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const int col = n0 + 8 * nt + t2;
            if (col >= vd) continue;
            store2(out + ((size_t)(first + t) * sh.nh + h) * vd + col, acc[nt][2 * r] * inv * sh.norm_w[col], acc[nt][2 * r + 1] * inv * sh.norm_w[col + 1]);
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
#define HK_RUN(T)                                                                                                      \
    do {                                                                                                               \
        const size_t kv_smem = (size_t)(3 + HkValues<T>::PLANES) * HK_C * HB_LD * 2 + (4 + HK_C) * HK_D * 4;            \
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
