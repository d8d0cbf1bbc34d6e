// Latent attention for prompt portions on the 5th-generation tensor cores (bfloat16), fed by TMA.
//
// The mathematics is that of latent_attention_mma.cu: the rows of a query tile are (token, head) pairs of one request in the
// order they lie in memory, all heads read the same cached rows [c | k_rot], and the values are the first kr numbers of the
// very rows that are the keys.  A tile is 128 such rows and up to 256 of the value columns (wider latents have
// their scores formed once per 256 columns: tensor memory has room for 256 columns of sums beside the scores).
//
// The query tile is kb blocks of [128][64], kb = (kr + rot) / 64 <= 9: the first two in tensor memory, the others in shared memory.
// A tile of 64 keys is kb blocks of [64][64], in groups of eight keys: the blocks that are only keys here, and the blocks that are this
// block's values, of which there are two buffers; 216 KB at kr 512, rot 64.  The key-only blocks may be refilled when the
// scores on them are complete, a buffer of values when its product is.
//   warps 4-7  copy the key-only blocks, every fourth group of eight keys each; warps 8, 9 the values.  A box holds eight keys of
//            several blocks
//   warp 10  products: the scores of the next tile (under the softmax of this one), then O += P V of this one
//   warps 0-3  softmax, a thread per row: S by tcgen05.ld, P = exp2(S - reference) back to tensor memory as bfloat16, the A
//            operand of O += P V; the reference moves, and O is rescaled, only when a row's maximum has grown by 2^8
// At the end the sink joins the denominator, the gate multiplies, and the row is stored.
//
// One block per SM walks through its tiles, so that a tile's queries and first keys come under the tile before and its results leave
// under the scores of the next.
//
// Measured on one B200, 16 heads, kr 512, rot 64, pages of 16, two prompts of 1000 tokens: 81 us (mma.sync kernel 251; 170 with one
// buffer of values, boxes of one block, products issued block by block under one lane, and a block per tile).  A tile of 64 keys
// takes 2600 clocks, 2250 of them products: 36 of 64 columns for the scores at 48 (the query tile's rows are read from shared memory
// each time; 32 from tensor memory), four of 256 for the values.  A query tile costs some 6000 beside its key tiles. Clock stamps:
// profiles/latent_attention_tc_clocks.md.
//
// Waits are bounded: one that expires marks the block dead, `status` gets 6, and the block waits (again with a limit) for its
// copies under way, frees its tensor memory and leaves.
#include "latent_attention.cuh"
#include "tcgen05.cuh"
#include "tma_host.h"

#define LT_KEY_COPIERS 4                // warps that issue copies of keys; two of values
#define LT_COPIERS (LT_KEY_COPIERS + 2)
#define LT_THREADS (128 + 32 * LT_COPIERS + 32)
#define LT_ROWS 128
#define LT_KEYS 64
#define LT_Q_BLK (LT_ROWS * 128u)       // bytes of one [rows][64] block
#define LT_K_BLK (LT_KEYS * 128u)
#define LT_MAX_BLOCKS 9
#define LT_Q_TMEM 2                     // blocks of the query tile in tensor memory (what O, S and P leave of it)
#define LT_LAZY 8.f

struct LatentTc {
    int kb, vb, vb_all;                 // blocks of 64: of a row, of this launch's value columns per block, of kr
    int max_pages, page_size, page_shift, n_seqs, nh, window, gate_ld, n_tiles, parts;
    float scale_log2;
    const int *positions, *q_start, *start_pos, *slots, *block_table;
    const float* sink;
    const bf16 *q, *gates;
    // boxes of a group of eight keys, for each part of the values, of its key-only blocks [0] and its values [1]: first block, and
    // 128 where the box has vb blocks and not one
    int n_boxes[2][2];
    unsigned char box[2][2][LT_MAX_BLOCKS];
};


// S (+)= query blocks FROM .. TO - 1 times a key tile's, whose descriptor `part` stands at block FROM (one thread issues)
template <int FROM, int TO>
__device__ __forceinline__ void lt_blocks(uint32_t d, uint32_t tq, uint64_t dq, uint64_t part, uint32_t idesc, bool fresh) {
#pragma unroll
    for (int k = FROM; k < TO; ++k)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const uint64_t db = part + (((k - FROM) * 1024 + kk * 32) >> 4);
            const int more = !(fresh && k == FROM && kk == 0);
            if (k < LT_Q_TMEM) tc_mma_ts(d, tq + 32 * k + 8 * kk, db, idesc, more);
            else tc_mma(d, dq + (((k - LT_Q_TMEM) * LT_Q_BLK + kk * 32) >> 4), db, idesc, more);
        }
}

// a query tile of this block
struct LatentTile {
    int tok0, n_rows, r0, start, slot;      // request: first token, rows, and position before it; first row of the tile
    int lo, hi;                             // keys lo .. hi - 1 are seen by some row of the tile
};

// KB, NV: blocks of a row and of a block's values where they are known when this is compiled, else 0.  A tile's scores are then
// issued in two runs with constant offsets; block by block they took 75 clocks a product to issue, 48 so (of 36 a tile).
template <int KB, int NV>
__global__ void __launch_bounds__(LT_THREADS, 1)
latent_attention_tc_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map,
                           const __grid_constant__ CUtensorMap k1_map, bf16* __restrict__ out, const __grid_constant__ LatentTc p,
                           int* status) {
    extern __shared__ unsigned char lt_raw[];
    __shared__ __align__(8) unsigned long long s_q, s_qt, s_keys, s_values[2], s_kfree[2], s_score[2], s_sum[2], s_p;      // [key tile & 1]
    __shared__ uint32_t s_tmem;
    __shared__ int s_dead, s_issued[LT_COPIERS], s_count;
    __shared__ LatentTile s_tiles[32];
    const uint32_t base = (tc_smem(lt_raw) + 1023u) & ~1023u;
    const int qt = min(LT_Q_TMEM, p.kb);
    const int tid = threadIdx.x, warp = tc_warp(), lane = tid & 31;
    volatile int* dead = &s_dead;
    ST_PDL_WAIT();
    if (warp == 0) {
        // This block's query tiles, a lane each (the launcher sees to it that there are no more).  The last tiles of a request have the
        // longest key ranges: first, all value columns of a tile in blocks side by side, and the blocks forwards and backwards in
        // turn, so that who has the longest of one round has the shortest of the next.
        const long long per_turn = gridDim.x / p.parts, at = blockIdx.x / p.parts;
        const long long place = lane * per_turn + (lane & 1 ? per_turn - 1 - at : at);
        LatentTile t;
        int left = place < p.n_tiles ? p.n_tiles - 1 - (int)place : 0x7fffffff, req = -1, from = p.q_start[0];
        t.tok0 = t.n_rows = 0;
#pragma unroll 8
        for (int i = 0; i < p.n_seqs; ++i) {
            const int to = p.q_start[i + 1], rows = (to - from) * p.nh, n = (rows + LT_ROWS - 1) / LT_ROWS;
            if (req < 0) {
                if (left < n) { req = i; t.tok0 = from; t.n_rows = rows; }
                else left -= n;
            }
            from = to;
        }
        const bool live = req >= 0 && p.positions[t.tok0] >= 0;      // (not padding of a fixed-shape step)
        if (live) {
            t.start = p.start_pos[req];
            t.slot = p.slots[req];
            t.r0 = left * LT_ROWS;
            t.hi = t.start + (min(t.r0 + LT_ROWS, t.n_rows) - 1) / p.nh + 1;
            t.lo = p.window > 0 ? max(0, t.start + t.r0 / p.nh - p.window + 1) : 0;
        }
        const uint32_t all = __ballot_sync(0xffffffffu, live);
        if (live) s_tiles[__popc(all & ((1u << lane) - 1))] = t;
        if (lane == 0) s_count = __popc(all);
    } else if (tid == 32) {
        tc_mbar_init(tc_smem(&s_q), LT_KEY_COPIERS);
        tc_mbar_init(tc_smem(&s_qt), 4);
        tc_mbar_init(tc_smem(&s_keys), LT_KEY_COPIERS);
        for (int i = 0; i < 2; ++i) tc_mbar_init(tc_smem(&s_values[i]), 2);
        for (int i = 0; i < 2; ++i) { tc_mbar_init(tc_smem(&s_kfree[i]), 1); tc_mbar_init(tc_smem(&s_score[i]), 1); tc_mbar_init(tc_smem(&s_sum[i]), 1); }
        tc_mbar_init(tc_smem(&s_p), 4);
        tc_mbar_init_fence();
        s_dead = 0;
        for (int i = 0; i < LT_COPIERS; ++i) s_issued[i] = 0;
    } else if (warp == 4 + LT_COPIERS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem(&s_tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    ST_PDL_TRIGGER();                                         // behind the allocation
    const uint32_t tmem = s_tmem;                             // O at 0 (64 vb columns), S at 256 and 320, P at 384 and 416, queries at 448
    const int n_mine = s_count;
    const int part = blockIdx.x % p.parts, v0 = part * p.vb, nv = min(p.vb, p.vb_all - v0);      // this block's values: blocks v0 .. v0 + nv - 1
    // key-only blocks: 0 .. v0 - 1 and v0 + nv .. kb - 1, nk of them; a group of eight keys is nk blocks of [8][64] in one place and nv in
    // another
    const int nk = p.kb - nv;
    const uint32_t k_grp = nk * 1024u, v_grp = nv * 1024u, v_buf = 8 * v_grp;
    const uint32_t sQ = base, sK = sQ + (p.kb - qt) * LT_Q_BLK, sV = sK + 8 * k_grp, sO = sV + 2 * v_buf;      // queries from block qt on
    // tile t and its key tiles
#define LT_TILE(t)                                                                                                     \
    const LatentTile T = s_tiles[t];                                                                                   \
    const int kt0 = T.lo / LT_KEYS, n_kt = (T.hi + LT_KEYS - 1) / LT_KEYS - kt0
    if (warp >= 4 && warp < 4 + LT_COPIERS) {
        // ---- copies.  A page without a key this query tile may see may have been given back: its rows (masked, and zeroed as
        // values) are filled from the tile's first live page.
        const int me = warp - 4, kind = me >= LT_KEY_COPIERS;                // kind 0: keys, 1: values
        const int step = kind ? 2 : LT_KEY_COPIERS, first_group = kind ? me - LT_KEY_COPIERS : me, groups = 8 / step;
        // This warp's boxes of a key tile: of its groups of eight keys (every step-th) the blocks in boxes of vb or of one.  Lane j has
        // the page of the j-th group.  Where the boxes are known when this is compiled they are issued with constant offsets; else
        // a lane has its own boxes, at most two, and knows all but the page before the key tiles begin.  (A tile's four boxes of a
        // key warp took 3500 clocks to issue with one lane working them out, 1400 with the whole warp doing so, 600 with a
        // lane for each.)
        const unsigned per_group = p.n_boxes[part][kind];
        int b_turn[2], b_row[2], b_from[2], b_big[2];
        uint32_t b_dst[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const unsigned e = lane + 32 * x;
            b_turn[x] = -1;
            b_row[x] = b_from[x] = b_big[x] = 0;
            b_dst[x] = 0;
            if (KB > 0 || e >= groups * per_group) continue;
            const int turn = e / per_group, grp = first_group + step * turn, box = p.box[part][kind][e - turn * per_group];
            b_from[x] = box & 127;
            b_big[x] = box >> 7;
            b_turn[x] = turn;
            b_row[x] = 8 * grp & (p.page_size - 1);
            b_dst[x] = kind ? sV + grp * v_grp + (b_from[x] - v0) * 1024 : sK + grp * k_grp + (b_from[x] < v0 ? b_from[x] : b_from[x] - nv) * 1024;
        }
        int g = 0;                                            // key tiles of this block so far: buffer g & 1, phase (g >> 1) & 1
        bool ok = true;
        for (int t = 0; t < n_mine && ok; ++t) {
            LT_TILE(t);
            const int* bt = p.block_table + (size_t)T.slot * p.max_pages;
            const int my_key = 8 * (first_group + step * min(lane, groups - 1));
            auto page_of = [&](int i) -> int {
                if (i >= n_kt) return 0;
                const int k0 = (kt0 + i) * LT_KEYS;
                const int first = max(k0, T.lo) >> p.page_shift, last = (min(k0 + LT_KEYS, T.hi) - 1) >> p.page_shift;
                return bt[min(max((k0 + my_key) >> p.page_shift, first), last)];
            };
            int page = page_of(0);
            // the key warps bring the queries as well: a warp's 32 rows of the blocks in tensor memory, and every fourth of the others
            uint32_t q[LT_Q_TMEM][32];
            if (kind == 0) {
                const int row = T.r0 + me * 32 + lane;
                const bool live = row < T.n_rows;
                const uint4* src = reinterpret_cast<const uint4*>(p.q + ((size_t)T.tok0 * p.nh + (live ? row : 0)) * (64 * p.kb));
#pragma unroll
                for (int k = 0; k < LT_Q_TMEM; ++k)
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const uint4 u = live && k < qt ? __ldcg(src + 8 * k + e) : make_uint4(0, 0, 0, 0);
                        q[k][4 * e] = u.x; q[k][4 * e + 1] = u.y; q[k][4 * e + 2] = u.z; q[k][4 * e + 3] = u.w;
                    }
            }
            for (int i = 0; i < n_kt; ++i, ++g) {
                const int next = page_of(i + 1);
                if (page < 0 && status) *status = 1;          // a hole: its rows read as zeros
                // The key-only blocks are free when the scores on them are complete, the queries when all scores are, a buffer of
                // values when the product of the key tile before the last one is.  (Barriers per buffer, and every phase is
                // waited for: a wait that finds two phases gone by sees the parity of none.)
                if (kind == 0 && g > 0) ok = tc_wait_warp(tc_smem(&s_kfree[0]) + 8 * ((g - 1) & 1), ((g - 1) >> 1) & 1, dead);
                if (kind == 1 && g > 1) ok = tc_wait_warp(tc_smem(&s_sum[0]) + 8 * (g & 1), ((g - 2) >> 1) & 1, dead);
                if (!ok) break;
                const uint32_t mb = kind ? tc_smem(&s_values[0]) + 8 * (g & 1) : tc_smem(&s_keys);
                if constexpr (KB > 0) {
                    int pg[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) pg[j] = __shfl_sync(0xffffffffu, page, j);
                    if (tc_elect()) {
                        tc_mbar_expect_tx(mb, (kind ? NV : KB - NV) * groups * 1024u);
                        s_issued[me] = g + 1;
                        if (kind == 0) {
#pragma unroll
                            for (int j = 0; j < 8 / LT_KEY_COPIERS; ++j) {
                                const uint32_t dst = sK + (first_group + j * LT_KEY_COPIERS) * ((KB - NV) * 1024u);
                                const int row = 8 * (first_group + j * LT_KEY_COPIERS) & (p.page_size - 1);
                                tc_tma_load_4d(dst, &k_map, 0, row, v0 == 0 ? NV : 0, pg[j], mb);
#pragma unroll
                                for (int k = 2 * NV; k < KB; ++k) tc_tma_load_4d(dst + (k - NV) * 1024, &k1_map, 0, row, k, pg[j], mb);
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                tc_tma_load_4d(sV + (g & 1) * v_buf + (first_group + 2 * j) * (NV * 1024u), &k_map, 0,
                                               8 * (first_group + 2 * j) & (p.page_size - 1), v0, pg[j], mb);
                        }
                    }
                    __syncwarp();
                } else {
                    if (lane == 0) {
                        if (per_group) tc_mbar_expect_tx(mb, (kind ? nv : nk) * groups * 1024u);
                        s_issued[me] = g + 1;
                    }
                    __syncwarp();
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        const int pg = __shfl_sync(0xffffffffu, page, max(b_turn[x], 0));
                        if (b_turn[x] >= 0)
                            tc_tma_load_4d(b_dst[x] + (kind ? (g & 1) * v_buf : 0), b_big[x] ? &k_map : &k1_map, 0, b_row[x], b_from[x], pg, mb);
                    }
                    __syncwarp();
                }
                page = next;
                if (kind == 0 && i == 0) {
                    // (the scores of g - 3 are complete since those on the keys of g - 1 are: this is the phase that is waited for)
                    if (g > 0) ok = tc_wait_warp(tc_smem(&s_score[0]) + 8 * ((g - 1) & 1), ((g - 1) >> 1) & 1, dead);
                    if (!ok) break;
                    tc_fence_after_sync();
                    if (tc_elect()) {
                        int n = 0;
                        for (int k = qt + me; k < p.kb; k += LT_KEY_COPIERS) ++n;
                        tc_mbar_expect_tx(tc_smem(&s_q), n * LT_Q_BLK);
                        for (int k = qt + me; k < p.kb; k += LT_KEY_COPIERS)
                            tc_tma_load_2d(sQ + (k - qt) * LT_Q_BLK, &q_map, k * 64, T.tok0 * p.nh + T.r0, tc_smem(&s_q));
                    }
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < LT_Q_TMEM; ++k)
                        if (k < qt) tc_st32(tmem + ((uint32_t)(me * 32) << 16) + 448 + 32 * k, reinterpret_cast<const float*>(q[k]));
                    tc_st_wait();
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc_smem(&s_qt)) : "memory");
                }
                __syncwarp();
            }
        }
    } else if (warp == 4 + LT_COPIERS) {
        // ---- products
        const uint32_t idesc_s = tc_idesc(LT_ROWS, LT_KEYS, 0, 0), idesc_o = tc_idesc(LT_ROWS, 64 * nv, 0, 1);
        const uint64_t dq = tc_desc(sQ, 16, 1024), dk = tc_desc(sK, 16, k_grp);
        int g0 = 0;
        bool ok = true;
        for (int t = 0; t < n_mine && ok; ++t) {
        LT_TILE(t);
        auto scores = [&](int g) -> bool {                    // S of key tile g into its buffer: key-only blocks, then values
            const uint32_t d = tmem + 256 + 64 * (g & 1);
            const uint64_t dv = tc_desc(sV + (g & 1) * v_buf, 16, v_grp);
            bool first = true;
            // block k of the queries against block `at` of a part
            auto block = [&](int k, uint64_t part, int at) {
                const uint64_t db = part + ((at * 1024) >> 4), da = dq + (((k - qt) * LT_Q_BLK) >> 4);
                const uint32_t ta = tmem + 448 + 32 * k;
                if (tc_elect()) {
                    if (k < qt) {
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) tc_mma_ts(d, ta + 8 * kk, db + ((kk * 32) >> 4), idesc_s, !first || kk > 0);
                    } else {
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) tc_mma(d, da + ((kk * 32) >> 4), db + ((kk * 32) >> 4), idesc_s, !first || kk > 0);
                    }
                }
                __syncwarp();
                first = false;
            };
            if (nk > 0) {
                if (!tc_wait_warp(tc_smem(&s_keys), g & 1, dead)) return false;
                tc_fence_after_sync();
                if constexpr (KB > 0) {
                    if (tc_elect()) {
                        if (v0 == 0) lt_blocks<NV, KB>(d, tmem + 448, dq, dk, idesc_s, true);
                        else {
                            lt_blocks<0, NV>(d, tmem + 448, dq, dk, idesc_s, true);
                            lt_blocks<2 * NV, KB>(d, tmem + 448, dq, dk + ((NV * 1024) >> 4), idesc_s, false);
                        }
                    }
                    __syncwarp();
                } else {
                    for (int k = 0; k < v0; ++k) block(k, dk, k);
                    for (int k = v0 + nv; k < p.kb; ++k) block(k, dk, k - nv);
                }
            }
            if (tc_elect()) tc_commit(tc_smem(&s_kfree[0]) + 8 * (g & 1));
            __syncwarp();
            if (!tc_wait_warp(tc_smem(&s_values[0]) + 8 * (g & 1), (g >> 1) & 1, dead)) return false;
            tc_fence_after_sync();
            if constexpr (KB > 0) {
                if (tc_elect()) {
                    if (v0 == 0) lt_blocks<0, NV>(d, tmem + 448, dq, dv, idesc_s, false);
                    else lt_blocks<NV, 2 * NV>(d, tmem + 448, dq, dv, idesc_s, false);
                    tc_commit(tc_smem(&s_score[0]) + 8 * (g & 1));
                }
                __syncwarp();
                return true;
            }
            for (int k = v0; k < v0 + nv; ++k) block(k, dv, k - v0);
            if (tc_elect()) tc_commit(tc_smem(&s_score[0]) + 8 * (g & 1));
            __syncwarp();
            return true;
        };
        ok = tc_wait_warp(tc_smem(&s_q), t & 1, dead) && tc_wait_warp(tc_smem(&s_qt), t & 1, dead);
        tc_fence_after_sync();
        ok = ok && scores(g0);
        for (int i = 0; i < n_kt && ok; ++i) {
            const int g = g0 + i;
            // (S's other buffer is free: the softmax threads had read it when they wrote P of the key tile before)
            if (i + 1 < n_kt) ok = scores(g + 1);
            if (ok) ok = tc_wait_warp(tc_smem(&s_p), g & 1, dead);         // P(g) is written, S(g) read, and O of the tile before
            if (!ok) break;
            tc_fence_after_sync();
            const uint64_t dv = tc_desc(sV + (g & 1) * v_buf, 1024, v_grp);
            if (tc_elect()) {
#pragma unroll
                for (int j = 0; j < LT_KEYS / 16; ++j)
                    tc_mma_ts(tmem, tmem + 384 + 32 * (g & 1) + j * 8, dv + ((j * 2 * v_grp) >> 4), idesc_o, i > 0 || j > 0);
                tc_commit(tc_smem(&s_sum[0]) + 8 * (g & 1));
            }
            __syncwarp();
        }
        g0 += n_kt;
        }
    } else if (warp < 4) {
        // ---- softmax: thread tid is row tid of the tile and lane tid of tensor memory
        const uint32_t t_row = tmem + ((uint32_t)(warp * 32) << 16);
        int g0 = 0;
        bool ok = true;                                       // the same in every lane of a warp
        for (int t = 0; t < n_mine && ok; ++t) {
        LT_TILE(t);
        const int lo = T.lo, hi = T.hi, row = T.r0 + tid, tok = row / p.nh;
        const bool live = row < T.n_rows;
        const int pos = live ? T.start + tok : -1, first_key = p.window > 0 ? pos - p.window + 1 : 0;
        float m_ref = -INFINITY, l_run = 0.f;
        for (int i = 0; i < n_kt && ok; ++i) {
            const int g = g0 + i;
            ok = tc_wait_warp(tc_smem(&s_score[0]) + 8 * (g & 1), (g >> 1) & 1, dead);
            if (!ok) break;
            tc_fence_after_sync();
            float s[LT_KEYS];
            tc_ld32(t_row + 256 + 64 * (g & 1), s);
            tc_ld32(t_row + 256 + 64 * (g & 1) + 32, s + 32);
            tc_ld_wait();
            const int k0 = (kt0 + i) * LT_KEYS;
            if (k0 + LT_KEYS - 1 > pos || k0 < first_key) {
#pragma unroll
                for (int c = 0; c < LT_KEYS; ++c)
                    if (k0 + c > pos || k0 + c < first_key) s[c] = -INFINITY;
            }
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < LT_KEYS; c += 8)
#pragma unroll
                for (int e = 0; e < 4; ++e) mx4[e] = tc_max3(mx4[e], s[c + 2 * e], s[c + 2 * e + 1]);
            const float m_new = fmaxf(m_ref, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2);
            const bool move = m_new > m_ref + LT_LAZY;
            const float corr = move ? tc_exp2(m_ref - m_new) : 1.f;
            if (move) m_ref = m_new;
            const float neg_m = m_ref == -INFINITY ? 0.f : -m_ref;
            float rs[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            uint32_t w[LT_KEYS / 2];
#pragma unroll
            for (int c = 0; c < LT_KEYS / 2; ++c) {
                float a0, a1;
                tc_fma2(a0, a1, s[2 * c], s[2 * c + 1], p.scale_log2, neg_m);
                const float p0 = tc_exp2(a0), p1 = tc_exp2(a1);
                tc_add2(rs[2 * (c & 3)], rs[2 * (c & 3) + 1], p0, p1);
                const __nv_bfloat162 pk = __floats2bfloat162_rn(p0, p1);
                w[c] = *reinterpret_cast<const uint32_t*>(&pk);
            }
            if (i > 0) {                                      // O += P V of the tile before: O may be rescaled after it
                ok = tc_wait_warp(tc_smem(&s_sum[0]) + 8 * ((g - 1) & 1), ((g - 1) >> 1) & 1, dead);
                if (!ok) break;
                tc_fence_after_sync();
                if (__any_sync(0xffffffffu, move)) {
                    for (int c = 0; c < 2 * nv; ++c) {
                        float o[32];
                        tc_ld32(t_row + c * 32, o);
                        tc_ld_wait();
#pragma unroll
                        for (int e = 0; e < 32; ++e) o[e] *= corr;
                        tc_st32(t_row + c * 32, o);
                    }
                    l_run *= corr;
                }
            }
            if (k0 < lo || k0 + LT_KEYS > hi) {
                // Rows of the tile that no row of the block sees hold what the pages hold there, behind a request's last token
                // what an earlier owner of the page left: zeros take their place, for a weight of zero times what is not
                // finite is not zero.  The boxes have landed (the scores are complete), and the next ones wait for O += P V.
                tc_wait_warp(tc_smem(&s_values[0]) + 8 * (g & 1), (g >> 1) & 1, dead);
                const int head = min(max(lo - k0, 0), LT_KEYS), tail = max(min(hi - k0, LT_KEYS), head);
                if (lane < nv * 8) {                          // a lane per 16 bytes of a row's values (nv <= 4), a warp per row
                    const uint32_t at = sV + (g & 1) * v_buf + lane / 8 * 1024 + lane % 8 * 16;
                    for (int key = warp; key < LT_KEYS; key += 4)
                        if (key < head || key >= tail)
                            asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};\n" ::"r"(at + key / 8 * v_grp + key % 8 * 128), "r"(0) : "memory");
                }
                tc_fence_async_smem();
            }
            tc_st32(t_row + 384 + 32 * (g & 1), reinterpret_cast<const float*>(w));
            l_run += ((rs[0] + rs[1]) + (rs[2] + rs[3])) + ((rs[4] + rs[5]) + (rs[6] + rs[7]));
            tc_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc_smem(&s_p)) : "memory");
        }
        g0 += n_kt;
        if (ok) ok = tc_wait_warp(tc_smem(&s_sum[0]) + 8 * ((g0 - 1) & 1), ((g0 - 1) >> 1) & 1, dead);
        tc_fence_after_sync();
        const int h = row % p.nh;
        float k = 0.f;
        if (live) {
            const float snk = p.sink ? p.sink[h] * 1.4426950408889634f : -INFINITY;
            const float mf = fmaxf(m_ref, snk);
            const float c = m_ref == -INFINITY ? 0.f : exp2f(m_ref - mf);
            const float den = l_run * c + (snk > -INFINITY ? exp2f(snk - mf) : 0.f);
            float gate = 1.f;
            if (p.gates) gate = 1.f / (1.f + expf(-load1_cg(p.gates + (size_t)(T.tok0 + tok) * p.gate_ld + h)));
            k = den > 0.f ? c * gate / den : 0.f;
        }
        if (ok) {
            // 32 columns of a warp's 32 rows at a time by way of shared memory: eight rows' 64 bytes are then stored together (straight
            // from the lanes of tensor memory, 16 bytes of 32 rows, it took 5900 clocks).  Pieces of 16 bytes are turned by the
            // row, so that eight rows' writes hit distinct banks.
            const uint32_t mine = sO + warp * 2048;
            const int n = min(32, T.n_rows - T.r0 - warp * 32);
            bf16* dst = out + ((size_t)T.tok0 * p.nh + T.r0 + warp * 32) * (64 * p.vb_all) + 64 * v0 + (lane & 3) * 8;
            for (int c = 0; c < 2 * nv; ++c) {
                float o[32];
                tc_ld32(t_row + c * 32, o);
                tc_ld_wait();
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    uint32_t w4[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const __nv_bfloat162 pk = __floats2bfloat162_rn(o[8 * e + 2 * j] * k, o[8 * e + 2 * j + 1] * k);
                        w4[j] = *reinterpret_cast<const uint32_t*>(&pk);
                    }
                    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(mine + lane * 64 + ((e ^ (lane >> 1 & 3)) << 4)),
                                 "r"(w4[0]), "r"(w4[1]), "r"(w4[2]), "r"(w4[3]) : "memory");
                }
                __syncwarp();
#pragma unroll
                for (int r0 = 0; r0 < 32; r0 += 8) {
                    const int r = r0 + (lane >> 2);
                    uint4 u;
                    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];\n" : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
                                 : "r"(mine + r * 64 + (((lane & 3) ^ (r >> 1 & 3)) << 4)) : "memory");
                    if (r < n) *reinterpret_cast<uint4*>(dst + (size_t)r * (64 * p.vb_all) + c * 32) = u;
                }
                __syncwarp();
            }
        }
        }
    }
#undef LT_TILE
    tc_fence_before_sync();
    __syncthreads();
    if (s_dead && tid == 0) {
        if (status) atomicExch(status, 6);
        int keys = s_issued[0];
        for (int i = 1; i < LT_KEY_COPIERS; ++i) keys = min(keys, s_issued[i]);
        const int values = min(s_issued[LT_KEY_COPIERS], s_issued[LT_KEY_COPIERS + 1]);
        if (keys) tc_wait(tc_smem(&s_keys), (keys - 1) & 1);
        for (int i = 0; i < 2; ++i) {
            const int n = (values + 1 - i) >> 1;              // key tiles that went to this buffer
            if (n) tc_wait(tc_smem(&s_values[i]), (n - 1) & 1);
        }
        for (int i = 0; i < 20000; ++i) __nanosleep(100);     // and by time the products, the queries, and copies that not all warps began
    }
    __syncthreads();
    if (warp == 4 + LT_COPIERS) {
        tc_fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512) : "memory");
    }
}

// Whether the kernel takes these sizes: latent and whole row in blocks of 64 columns, at most 512 and 576, pages of 8 to 64
// positions (a power of two).
ST_EXPORT int st_latent_attention_tc_applies(int kr, int rot, int page_size) {
    return kr > 0 && rot >= 0 && kr % 64 == 0 && rot % 64 == 0 && kr <= 512 && (kr + rot) / 64 <= LT_MAX_BLOCKS &&
           (page_size == 8 || page_size == 16 || page_size == 32 || page_size == 64);
}

// Blocks a step of n_tokens tokens gives (for the rule of who takes it).
ST_EXPORT int st_latent_attention_tc_blocks(int n_tokens, int nh, int kr) {
    return (int)(((long long)n_tokens * nh + LT_ROWS - 1) / LT_ROWS * ((kr / 64 + 3) / 4));
}

// Arguments as st_latent_attention_mma without parts of key ranges; n_pages: pages of the pool.
ST_EXPORT int st_latent_attention_tc(const void* q_lat, const void* pool, long long n_pages, long long page_stride,
                                     long long entry_offset, void* out, const int* positions, const int* q_start,
                                     const int* start_pos, const int* slots, const int* block_table, int max_pages, int n_tokens,
                                     int n_seqs, int nh, int kr, int rot, int page_size, const float* sink, const void* gates,
                                     int gate_ld, float scale, int* status, void* stream, int window) {
    if (n_tokens <= 0 || n_seqs <= 0) return 0;
    if (!st_latent_attention_tc_applies(kr, rot, page_size) || page_stride % 8 || entry_offset % 8) return ST_ERR_BAD_SIZE;
    if (nh <= 0 || n_pages <= 0 || !status || !aligned16(q_lat) || !aligned16(out) || !aligned16((const bf16*)pool + entry_offset))
        return ST_ERR_BAD_ARG;
    const int kd = kr + rot;
    const long long tiles = ((long long)n_tokens * nh + LT_ROWS - 1) / LT_ROWS + n_seqs;
    if (tiles * ((kr / 64 + 3) / 4) > 0x7fffffffLL || (long long)n_tokens * nh > 0x7fffffffLL || n_pages > 0x7fffffffLL) return ST_ERR_TOO_LARGE;
    const unsigned long long qd[2] = {(unsigned long long)kd, (unsigned long long)n_tokens * nh};
    const unsigned qb[2] = {64, LT_ROWS};
    LatentTc p;
    p.kb = kd / 64; p.vb_all = kr / 64;
    const int parts = p.parts = (p.vb_all + 3) / 4;
    p.vb = (p.vb_all + parts - 1) / parts;
    // a row's blocks of 64 columns are a dimension of their own, so that one box holds eight keys of several blocks
    const unsigned long long kdim[4] = {64, (unsigned long long)page_size, (unsigned long long)p.kb, (unsigned long long)n_pages};
    const unsigned long long kst[3] = {(unsigned long long)kd * 2, 128, (unsigned long long)page_stride * 2};
    const unsigned kb[4] = {64, 8, (unsigned)p.vb, 1}, k1b[4] = {64, 8, 1, 1};
    CUtensorMap q_map, k_map, k1_map;
    if (st_tma_encode_bf16(&q_map, q_lat, 2, qd, qb) ||
        st_tma_encode_bf16_strided(&k_map, (const bf16*)pool + entry_offset, 4, kdim, kst, kb) ||
        st_tma_encode_bf16_strided(&k1_map, (const bf16*)pool + entry_offset, 4, kdim, kst, k1b)) return ST_ERR_BAD_ARG;
    p.page_shift = 0;
    while ((1 << p.page_shift) < page_size) ++p.page_shift;
    for (int part = 0; part < parts; ++part)
        for (int kind = 0; kind < 2; ++kind) {
            const int v0 = part * p.vb, nv = p.vb < p.vb_all - v0 ? p.vb : p.vb_all - v0;
            const int runs[2][2] = {{kind ? v0 : 0, kind ? v0 + nv : v0}, {v0 + nv, kind ? v0 + nv : p.kb}};
            int n = 0;
            for (int r = 0; r < 2; ++r)
                for (int at = runs[r][0]; at < runs[r][1];) {
                    const bool big = at + p.vb <= runs[r][1];
                    p.box[part][kind][n++] = (unsigned char)(at | (big ? 128 : 0));
                    at += big ? p.vb : 1;
                }
            p.n_boxes[part][kind] = n;
        }
    p.max_pages = max_pages; p.page_size = page_size; p.n_seqs = n_seqs; p.nh = nh; p.window = window; p.gate_ld = gate_ld;
    p.n_tiles = (int)tiles; p.scale_log2 = scale * 1.4426950408889634f;
    p.positions = positions; p.q_start = q_start; p.start_pos = start_pos; p.slots = slots; p.block_table = block_table;
    p.sink = sink; p.gates = (const bf16*)gates; p.q = (const bf16*)q_lat;
    const size_t smem = (size_t)(p.kb > LT_Q_TMEM ? p.kb - LT_Q_TMEM : 0) * LT_Q_BLK + (size_t)(p.kb + p.vb) * LT_K_BLK + 4 * 2048 + 1024;
    // one block per SM, but at most 32 tiles a block
    long long per_turn = st_sm_count() / parts;
    if (per_turn < 1) per_turn = 1;
    if (per_turn > tiles) per_turn = tiles;
    if (per_turn * 32 < tiles) per_turn = (tiles + 31) / 32;
    const long long grid = per_turn * parts;
    auto launch = [&](auto kernel) -> int {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        return st_launch_pdl("latent_tc", kernel, dim3((unsigned)grid), dim3(LT_THREADS), smem, (cudaStream_t)stream, q_map, k_map,
                             k1_map, (bf16*)out, p, status);
    };
    if (kr == 512 && rot == 64) return launch(latent_attention_tc_kernel<9, 4>);
    return launch(latent_attention_tc_kernel<0, 0>);
}
