// The 32-bit matrix product for few rows (decode steps): see gemm_f32.cuh for the arithmetic.
//
// A tile is 16 rows of w and up to 8 or 16 of a, so that there are tiles for every SM; blocks walk through the tiles, and their warps take
// every WARPS-th group of 64 k each.  A warp copies its groups of w and a by 16-byte asynchronous copies into a ring of its own (64 KB of
// w under way per block, on into the next tile) and reads them back as fragments of mma.sync: a lane takes the four neighbours
// 4 t .. 4 t + 3 of rows g and g + 8 per step of 16 k, so a step's sixteen products are those of sixteen k in another order, which changes no
// bit.  The groups' sums meet in shared memory (two rounds of them, so that one is added up while the next is written), where the
// last four warps, which have the fewest groups, add them up in ascending order.
//
// Bound by instructions (1 x 2048 x 50272 before what follows: 65 % of the issue slots in use, DRAM 48 %), most of them cutting w and a
// into parts; so the copies' addresses go on by constant steps, and rows of a that are not there are not copied.  us on one B200, recorded calls over weights that are not in cache, in brackets addresses worked out copy by copy and every row
// copied, then float multiply-adds: 1 x 2048 x 8192 19.3 (21.2; 17.7), 1 x 4096 x 4096 18.8 (20.5; 19.7), 8 x 4096 x 4096 20.1 (20.5; 24.9),
// 16 x 768 x 3072 8.4 (11.0; 9.0), 16 x 2048 x 2048 10.5 (11.2; 13.7), 1 x 64 x 64 3.2 (3.3; 2.3).
#include "gemm_f32.cuh"
#include "mma_sync.cuh"

// NB: blocks of eight rows of a
template <int NB>
struct GemmFew {
    static constexpr int WARPS = NB == 1 ? 8 : 10, STAGES = 2;
    static constexpr int ROUND = 2 * WARPS;                  // groups whose sums are added up at a time
    static constexpr int ROWS = 16 + 8 * NB;                 // of a stage: w's, then a's, 256 bytes each
    static constexpr size_t SMEM = (size_t)WARPS * STAGES * ROWS * 256 + (size_t)2 * ROUND * NB * 128 * 4;
};

// 16-byte piece c of row r of a stage: odd rows turned by four pieces, so that the rows of a read's quarter hit distinct banks
__device__ __forceinline__ int gq_at(int r, int c) { return r * 64 + ((c ^ ((r & 1) << 2)) << 2); }

// a chain over k, left as soon as it is no number (it stays none)
__device__ __noinline__ float gq_chain(const float* a, const float* w, int k_dim) {
    float s = 0.f;
    int k = 0;
    for (; k + 8 <= k_dim && s == s; k += 8) {
        float x[8], y[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) { x[j] = __ldg(a + k + j); y[j] = __ldg(w + k + j); }
#pragma unroll
        for (int j = 0; j < 8; ++j) s = fmaf(x[j], y[j], s);
    }
    for (; k < k_dim && s == s; ++k) s = fmaf(__ldg(a + k), __ldg(w + k), s);
    return s;
}
// scale, bias, activation and store of one output; a sum that is not finite gives way to the chain
__device__ __forceinline__ void gq_store(const GemmF32& p, int row, int col, float v, float bias) {
    if (!(fabsf(v) < INFINITY)) v = gq_chain(p.a + (size_t)row * p.k_dim, p.w + (size_t)col * p.k_dim, p.k_dim);
    else v *= GF_DOWN2;
    p.out[(size_t)row * p.n_out + col] = gf_finish(p, v, bias);
}

template <int NB>
__global__ void __launch_bounds__(32 * GemmFew<NB>::WARPS, NB == 1 ? 2 : 1)
gemm_f32_few_kernel(const GemmF32 p, int tiles, int row_tiles, int vec_a, int vec_w) {
    using S = GemmFew<NB>;
    extern __shared__ __align__(16) float gq_smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    float* ring = gq_smem + warp * S::STAGES * S::ROWS * 64;
    float* sums = gq_smem + S::WARPS * S::STAGES * S::ROWS * 64;             // [round's parity][group][NB][row of a][row of w]
    const int out_of = tid - 32 * (S::WARPS - 4);                          // the last four warps add up: they have the fewest groups
    const int n_groups = (p.k_dim + GF_BK - 1) / GF_BK;
    // a lane's pieces: 16 bytes of every second row of w and of a
    const int c = lane & 15, odd_row = lane >> 4;
    const uint32_t ring_at = (uint32_t)__cvta_generic_to_shared(ring + gq_at(odd_row, c));
    const size_t two_rows = (size_t)2 * p.k_dim;
    auto first_of = [&](int tile) { return min(tile / row_tiles * 16, max(p.n_out - 16, 0)); };      // a last tile begins inside the one before
    auto copy = [&](int tile, int group, int stage) {
        const int k = group * GF_BK + 4 * c, m0 = first_of(tile), n0 = tile % row_tiles * (8 * NB);
        if (vec_a && vec_w && p.n_out >= 16) {
            // rows of a that are not there are not copied, or the last one in their place: what they give is not stored
            const bool on = k < p.k_dim;
            const uint32_t dst = ring_at + stage * (S::ROWS * 256);
            const float* src = on ? p.w + (size_t)(m0 + odd_row) * p.k_dim + k : p.w;
            const size_t step = on ? two_rows : 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) cp_async16_s(dst + i * 512, src + i * step, on);
#pragma unroll
            for (int i = 0; i < 4 * NB; ++i)
                if (n0 + 2 * i < p.n_rows)
                    cp_async16_s(dst + (8 + i) * 512, on ? p.a + (size_t)min(n0 + 2 * i + odd_row, p.n_rows - 1) * p.k_dim + k : p.a, on);
            return;
        }
        float* dst = ring + stage * S::ROWS * 64;
#pragma unroll 1                                             // (short code: unrolled by four it made the other path 4 % slower)
        for (int i = 0; i < S::ROWS / 2; ++i) {
            const int r = 2 * i + odd_row;
            const bool is_w = i < 8;
            const int row = is_w ? m0 + r : n0 + r - 16, rows = is_w ? p.n_out : p.n_rows;
            const float* src = (is_w ? p.w : p.a) + (size_t)(row < rows ? row : 0) * p.k_dim + k;
            float* at = dst + gq_at(r, c);
            if (is_w ? vec_w : vec_a) {
                const bool on = row < rows && k < p.k_dim;
                cp_async16(at, on ? src : is_w ? p.w : p.a, on);
                continue;
            }
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row < rows) {
                if (k < p.k_dim) v.x = __ldg(src);
                if (k + 1 < p.k_dim) v.y = __ldg(src + 1);
                if (k + 2 < p.k_dim) v.z = __ldg(src + 2);
                if (k + 3 < p.k_dim) v.w = __ldg(src + 3);
            }
            store4(at, v);
        }
    };
    int next_tile = warp < n_groups ? (int)blockIdx.x : tiles, next_group = warp;          // what this warp copies next
    auto fetch = [&](int stage) {
        if (next_tile < tiles) {
            copy(next_tile, next_group, stage);
            next_group += S::WARPS;
            if (next_group >= n_groups) { next_group = warp; next_tile += gridDim.x; }
        }
        cp_async_commit();
    };
#pragma unroll
    for (int s = 0; s < S::STAGES; ++s) fetch(s);
    int stage = 0, parity = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        float total[NB];                                     // outputs out_of of 128, block by block of rows
#pragma unroll
        for (int b = 0; b < NB; ++b) total[b] = 0.f;
        for (int round = 0; round < n_groups; round += S::ROUND, parity ^= 1) {
            const int end = min(n_groups, round + S::ROUND);
            float* part = sums + parity * S::ROUND * NB * 128;
            for (int group = round + warp; group < end; group += S::WARPS) {
                cp_async_wait<S::STAGES - 1>();
                __syncwarp();
                const float* src = ring + stage * S::ROWS * 64;
                uint32_t wh[4][4], wm[4][4], wl[4][4];       // [step of 16 k][fragment register]
                uint32_t ah[NB][4][2], am[NB][4][2], al[NB][4][2];
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const float4 v = load4(src + gq_at(g + 8 * r, 4 * kk + t));
                        gf_split(v.x, v.y, wh[kk][r], wm[kk][r], wl[kk][r]);
                        gf_split(v.z, v.w, wh[kk][2 + r], wm[kk][2 + r], wl[kk][2 + r]);
                    }
#pragma unroll
                    for (int b = 0; b < NB; ++b) {
                        const float4 v = load4(src + gq_at(16 + 8 * b + g, 4 * kk + t));
                        gf_split(v.x, v.y, ah[b][kk][0], am[b][kk][0], al[b][kk][0]);
                        gf_split(v.z, v.w, ah[b][kk][1], am[b][kk][1], al[b][kk][1]);
                    }
                }
                __syncwarp();
                fetch(stage);                                // the stage is read: the group but one takes its place
                float c[NB][4];
#pragma unroll
                for (int b = 0; b < NB; ++b) c[b][0] = c[b][1] = c[b][2] = c[b][3] = 0.f;
#define GQ_PRODUCT(W, A)                                                                                   \
    _Pragma("unroll") for (int kk = 0; kk < 4; ++kk)                                                       \
        _Pragma("unroll") for (int b = 0; b < NB; ++b) mma_bf16(c[b], W[kk], A[b][kk][0], A[b][kk][1])
                GQ_PRODUCT(wl, ah);
                GQ_PRODUCT(wh, al);
                GQ_PRODUCT(wm, am);
                GQ_PRODUCT(wm, ah);
                GQ_PRODUCT(wh, am);
                GQ_PRODUCT(wh, ah);
#undef GQ_PRODUCT
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    float* dst = part + ((group - round) * NB + b) * 128;
                    dst[2 * t * 16 + g] = c[b][0];
                    dst[(2 * t + 1) * 16 + g] = c[b][1];
                    dst[2 * t * 16 + g + 8] = c[b][2];
                    dst[(2 * t + 1) * 16 + g + 8] = c[b][3];
                }
                if (++stage == S::STAGES) stage = 0;
            }
            __syncthreads();                                 // (a round further on the same place is written again: behind the next one)
            if (out_of >= 0) {
#pragma unroll
                for (int b = 0; b < NB; ++b)
#pragma unroll 16
                    for (int i = 0; i < end - round; ++i) total[b] += part[(i * NB + b) * 128 + out_of];
            }
        }
        const int col = first_of(tile) + (out_of & 15), n0 = tile % row_tiles * (8 * NB);
        if (out_of >= 0 && col >= tile / row_tiles * 16 && col < p.n_out) {
            const float bias = p.bias ? __ldg(p.bias + col) : 0.f;
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                const int row = n0 + 8 * b + (out_of >> 4);
                if (row < p.n_rows) gq_store(p, row, col, total[b], bias);
            }
        }
    }
    cp_async_wait<0>();
}

template <int NB>
static int gq_launch(const GemmF32& p, cudaStream_t s) {
    using S = GemmFew<NB>;
    const int vec_a = p.k_dim % 4 == 0 && aligned16(p.a), vec_w = p.k_dim % 4 == 0 && aligned16(p.w);
    const cudaError_t e = cudaFuncSetAttribute(gemm_f32_few_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
    if (e != cudaSuccess) return (int)e;
    const int row_tiles = (p.n_rows + 8 * NB - 1) / (8 * NB);
    const long long all = ((long long)p.n_out + 15) / 16 * row_tiles;
    if (all > 0x3fffffffLL) return ST_ERR_TOO_LARGE;
    const int tiles = (int)all, most = (NB == 1 ? 2 : 1) * st_sm_count();
    gemm_f32_few_kernel<NB><<<tiles < most ? tiles : most, 32 * S::WARPS, S::SMEM, s>>>(p, tiles, row_tiles, vec_a, vec_w);
    return st_launch_status();
}

// Which tiles, and what they take, in units of 10 ns (one B200, recorded calls over weights that are not in cache): 8 rows 250, and 15 per
// group and 30 beside them for each tile an SM has, at least 18 per group; 16 rows 330, and 25 per group and 50 beside them for each round
// of tiles; four times as much where rows are not whole pieces of 16 bytes (40 x 770 x 2304 45 us).  us, tiles of 8 rows / 16 rows:
// 16 x 768 x 3072 8.4 / 10.7, 16 x 2048 x 2048 10.7 / 11.6, 16 x 8192 x 2048 36.1 / 34.8, 24 x 2048 x 2048 15.8 / 20.0, 24 x 768 x 768 5.1 / 6.7
static long long gq_cost(const GemmF32& p, int rows) {
    const long long tiles = ((long long)p.n_out + 15) / 16 * (((long long)p.n_rows + rows - 1) / rows), sms = st_sm_count();
    const long long n_groups = ((long long)p.k_dim + GF_BK - 1) / GF_BK;
    const long long slow = p.k_dim % 4 ? 4 : 1, per_tile = n_groups > 6 ? n_groups : 6;          // (a tile of few groups leaves warps idle)
    if (rows == 16) return 330 + slow * ((tiles + sms - 1) / sms) * (25 * per_tile + 50);
    const long long cost = tiles * (15 * per_tile + 30) / sms, least = 18 * n_groups;
    return 250 + slow * (cost < least ? least : cost);
}
long long gf_few_cost(const GemmF32& p, int& form) {
    const long long c8 = gq_cost(p, 8), c16 = gq_cost(p, 16);
    form = p.n_rows <= 8 || c8 < c16 ? -8 : -16;
    return form == -8 ? c8 : c16;
}
int gf_few_launch(const GemmF32& p, int rows, cudaStream_t s) {
    return rows == 8 ? gq_launch<1>(p, s) : gq_launch<2>(p, s);
}

// ---- k below GF_SHORT: a thread has a row of w and takes `rows` rows of a, one chain each.  Bound by the launch and, for many rows, by
// the results' way to memory.
__global__ void __launch_bounds__(256) gemm_f32_short_kernel(const GemmF32 p, int rows) {
    const int col = blockIdx.x * 256 + threadIdx.x;
    if (col >= p.n_out) return;
    float w[GF_SHORT - 1];
#pragma unroll
    for (int k = 0; k < GF_SHORT - 1; ++k) w[k] = k < p.k_dim ? __ldg(p.w + (size_t)col * p.k_dim + k) : 0.f;
    const float bias = p.bias ? __ldg(p.bias + col) : 0.f;
    for (long long row0 = (long long)blockIdx.y * rows; row0 < p.n_rows; row0 += (long long)gridDim.y * rows)
#pragma unroll 4
        for (int row = (int)row0; row < (row0 + rows < p.n_rows ? row0 + rows : p.n_rows); ++row) {
            const float* a = p.a + (size_t)row * p.k_dim;
            float s = 0.f;
#pragma unroll
            for (int k = 0; k < GF_SHORT - 1; ++k)
                if (k < p.k_dim) s = fmaf(__ldg(a + k), w[k], s);
            p.out[(size_t)row * p.n_out + col] = gf_finish(p, s, bias);
        }
}
int gf_short_launch(const GemmF32& p, cudaStream_t s) {
    const long long across = (p.n_out + 255LL) / 256;
    const int rows = across * p.n_rows > 8 * st_sm_count() ? 8 : 1;
    const long long down = (p.n_rows + rows - 1LL) / rows;
    gemm_f32_short_kernel<<<dim3((unsigned)across, (unsigned)(down < 65535 ? down : 65535)), 256, 0, s>>>(p, rows);
    return st_launch_status();
}
