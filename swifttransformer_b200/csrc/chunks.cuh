// Pieces of the recurrences that run long portions in chunks of 64 tokens side by side (hgrn2_chunks.cu, delta_chunks.cu).
#pragma once
#include "common.cuh"

#define HK_C 64            // tokens of a chunk
#define HK_H 32            // half of it
#define HK_D 128           // the most channels and values per head
#define HK_LD (HK_D + 4)
#define HK_LA (HK_C + 4)

// Requests with portions of at least `from` tokens run in chunks, the others walk: each by its own length, whoever shares the
// step.  A request's chunks have the places hk_place + 0, 1, ..: no two requests' overlap (a portion of `from` tokens and more
// moves both terms on), and hk_places hold all L = min(n_seqs, n / from) of them.
__host__ __device__ __forceinline__ int hk_place(int begin, int b, int from) {
    return begin / HK_C + (b == 0 ? 0 : b < begin / from ? b : begin / from);
}
static inline long long hk_places(int n_tokens, int L) { return ((long long)n_tokens + HK_C - 1) / HK_C + L - 1; }
static inline int hk_longs(int n_tokens, int n_seqs, int from) { return n_seqs < n_tokens / from ? n_seqs : n_tokens / from; }
// The chunk at `place`: false when none stands there.
__device__ __forceinline__ bool hk_find(const int* q_start, const int* positions, int n_seqs, int from, int place, int& b, int& first, int& n) {
    int lo = 0, hi = n_seqs;                              // the last request whose places begin at or before this one
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (hk_place(q_start[mid], mid, from) <= place) lo = mid; else hi = mid;
    }
    b = lo;
    const int begin = q_start[b], end = q_start[b + 1];
    const int chunk = place - hk_place(begin, b, from);
    first = begin + chunk * HK_C;
    n = min(HK_C, end - first);
    return chunk >= 0 && n > 0 && end - begin >= from && positions[begin] >= 0;      // (padding stands at position -1)
}

// 1 / d and z / d for d >= 1 (infinity among them), to the last bit or next to it: the hardware's reciprocal and one step of Newton's iteration
// for it, r + r (1 - d r); the quotient q = z r with its residual, q + r (z - q d) (P. W. Markstein, "Computation of elementary functions
// on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34 (1990)).  A thread's quotients so run side by side; as divisions they ran one
// after the other, some 360 clocks each: 32 of them were most of a chunk's time.
__device__ __forceinline__ float hk_inverse(float d) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d * 0.0625f));
    r *= 0.0625f;                                         // (from 2^126 on not normal, zero for an infinite d)
    return fmaf(r, fmaf(-fminf(d, 3.4028234e38f), r, 1.f), r);
}
__device__ __forceinline__ float hk_sigmoid(float z) { return hk_inverse(1.f + expf(-z)); }
__device__ __forceinline__ float hk_silu(float z) {
    const float d = 1.f + expf(-z), r = hk_inverse(d), q = z * r, rest = fmaf(-q, d, z);
    return rest < 0.f || rest > 0.f ? fmaf(rest, r, q) : q;          // (an infinite z or d has no residual)
}
// 1 / sqrt(x): the hardware's and a Newton step
__device__ __forceinline__ float hk_rsqrt(float x) {
    const float r = rsqrtf(x);
    return x > 1e-30f && x < 1e30f ? fmaf(0.5f * r, fmaf(-x * r, r, 1.f), r) : r;
}

__device__ __forceinline__ void hk_cp16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}

// The outputs of a chunk before their norm: acc[r][j] += rows row0 + 4 r, values col + 32 j .. + 3 of X S + A V, by 256 threads
// of 4 tokens x 8 values; X [HK_C][HK_LD], A [HK_C][HK_LA] (above its diagonal not read), V [HK_C][HK_LD] in shared memory, the
// state's rows S [dim][vd] from memory 16 at a time through the two stages `ring`, the first two of which the caller has
// asked for (hk_copy_rows) after anything else it copied.
#define HK_SR 16
__device__ __forceinline__ void hk_copy_rows(float* ring, const float* S, int i0, int dim, int vd) {
    float* dst = ring + ((i0 / HK_SR) & 1) * HK_SR * HK_LD;
    for (int i = threadIdx.x; i < HK_SR * (HK_D / 4); i += 256) {
        const int r = i / (HK_D / 4), c = (i % (HK_D / 4)) * 4;
        if (i0 + r < dim && c < vd) hk_cp16(dst + r * HK_LD + c, S + (size_t)(i0 + r) * vd + c);
    }
    asm volatile("cp.async.commit_group;\n" ::);
}
__device__ __forceinline__ float4 hk_fma4x4(float4 x, float4 y, float4 a) {
    return make_float4(fmaf(x.x, y.x, a.x), fmaf(x.y, y.y, a.y), fmaf(x.z, y.z, a.z), fmaf(x.w, y.w, a.w));
}
__device__ __forceinline__ void hk_fma4(float x, float4 v, float4& a) {
    a.x = fmaf(x, v.x, a.x); a.y = fmaf(x, v.y, a.y); a.z = fmaf(x, v.z, a.z); a.w = fmaf(x, v.w, a.w);
}
// acc += X[rows][0 .. 15] Y[0 .. 15][values]; the sixteen are added up by themselves first (a chain of 192 additions in a row
// costs half again as much accuracy as the walk over the tokens has)
__device__ __forceinline__ void hk_sixteen(float4 (&acc)[4][2], const float* X, int ldx, const float* Y, int steps) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        float4 part[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) part[r] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
            if (i >= steps) break;
            const float* y = Y + i * HK_LD + 32 * j;
            const float4 y0 = load4(y), y1 = load4(y + HK_LD), y2 = load4(y + 2 * HK_LD), y3 = load4(y + 3 * HK_LD);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float4 x = load4(X + 4 * r * ldx + i);
                hk_fma4(x.x, y0, part[r]); hk_fma4(x.y, y1, part[r]); hk_fma4(x.z, y2, part[r]); hk_fma4(x.w, y3, part[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r][j] = add4(acc[r][j], part[r]);
    }
}
// The same of the sixteen tokens that hold the rows themselves: row rl + 4 r adds the tokens up to itself and meets no later
// one, whatever its values are (a weight of zero times a number that is not finite is not zero).
__device__ __forceinline__ void hk_own_sixteen(float4 (&acc)[4][2], const float* A, const float* V, int rl) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        float4 part[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) part[r] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float* y = V + 4 * i * HK_LD + 32 * j;
            const float4 y0 = load4(y), y1 = load4(y + HK_LD), y2 = load4(y + 2 * HK_LD), y3 = load4(y + 3 * HK_LD);
#pragma unroll
            for (int r = i; r < 4; ++r) {
                const float4 x = load4(A + 4 * r * HK_LA + 4 * i);
                hk_fma4(x.x, y0, part[r]);
                if (r > i || rl >= 1) hk_fma4(x.y, y1, part[r]);
                if (r > i || rl >= 2) hk_fma4(x.z, y2, part[r]);
                if (r > i || rl >= 3) hk_fma4(x.w, y3, part[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r][j] = add4(acc[r][j], part[r]);
    }
}
__device__ __forceinline__ void hk_outputs(float4 (&acc)[4][2], const float* X, const float* A, const float* V, float* ring,
                                           const float* S, int n, int dim, int vd, int row0, int col) {
    const int warp = threadIdx.x >> 5;
    const bool active = (warp & 1) * 64 < vd && (warp >> 1) * 16 < n;
    for (int i0 = 0; i0 < dim; i0 += HK_SR) {
        asm volatile("cp.async.wait_group 1;\n" ::);
        __syncthreads();
        if (active)
            hk_sixteen(acc, X + row0 * HK_LD + i0, HK_LD, ring + ((i0 / HK_SR) & 1) * HK_SR * HK_LD + col, dim - i0);
        __syncthreads();
        if (i0 + 2 * HK_SR < dim) hk_copy_rows(ring, S, i0 + 2 * HK_SR, dim, vd);
        else asm volatile("cp.async.commit_group;\n" ::);
    }
    if (active) {
        const int s0 = (warp >> 1) * 16;                      // the sixteen tokens of the warp's own rows
        for (int s = 0; s < s0; s += 16) hk_sixteen(acc, A + row0 * HK_LA + s, HK_LA, V + s * HK_LD + col, 16);
        hk_own_sixteen(acc, A + row0 * HK_LA + s0, V + s0 * HK_LD + col, row0 - s0);
    }
}
