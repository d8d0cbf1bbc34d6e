// Latent attention for prompt portions on the 5th-generation tensor cores (bfloat16), fed by TMA.
//
// The mathematics is that of latent_attention_mma.cu: the rows of a query tile are (token, head) pairs of one request in the
// order they lie in memory, all heads read the same cached rows [c | k_rot], and the values are the first kr numbers of the
// very rows that are the keys.  A block serves 128 such rows and up to 256 of the value columns (wider latents have
// their scores formed once per 256 columns: tensor memory has room for 256 columns of sums beside the scores).
//
// Shared memory holds the query tile (kb blocks of [128][64], kb = (kr + rot) / 64 <= 9) and one tile of 64 keys (kb
// blocks of [64][64]), 216 KB at kr 512, rot 64.  There is no room for a second key tile, so a tile comes in two parts of their
// own barriers: the blocks that are only keys may be refilled when the scores are complete, the blocks that are this block's values
// when their product is.
//   warps 4-7  copies: the query blocks, then per key tile the two parts, every fourth page each
//   warp 8   products: O += P V of a tile, then the scores of the next one, key-only blocks first (under the values' copies)
//   warps 0-3  softmax, a thread per row: S by tcgen05.ld, P = exp2(S - reference) back to tensor memory as bfloat16, the A
//            operand of O += P V; the reference moves, and O is rescaled, only when a row's maximum has grown by 2^8
// At the end the sink joins the denominator, the gate multiplies, and the row is stored.
//
// Measured on one B200, 16 heads, kr 512, rot 64, pages of 16: two prompts of 1000 tokens 171 us (mma.sync kernel 251; 168
// without the rows cleared in a block's last tile), one of 700 58 (86), 450 tokens behind 1200 120 (184).  A tile of 64 keys
// takes about 7300 clocks (by clock stamps in a copy of the kernel): 2050 for the key-only blocks' copies (under the softmax of
// the tile before), 2900 for the values', 2150 for the scores on them, 1400 for the softmax: a product of 64 columns takes as
// long as one of 256, about 130 clocks per 16 dimensions, for its rows of the query tile are read each time.
//
// Waits are bounded: one that expires marks the block dead, `status` gets 6, and the block waits (again with a limit) for its
// copies under way, frees its tensor memory and leaves.
#include "latent_attention.cuh"
#include "tcgen05.cuh"
#include "tma_host.h"

#define LT_COPIERS 4                    // warps that issue copies
#define LT_THREADS (128 + 32 * LT_COPIERS + 32)
#define LT_ROWS 128
#define LT_KEYS 64
#define LT_Q_BLK (LT_ROWS * 128u)       // bytes of one [rows][64] block
#define LT_K_BLK (LT_KEYS * 128u)
#define LT_MAX_BLOCKS 9
#define LT_LAZY 8.f

struct LatentTc {
    int kb, vb, vb_all;                 // blocks of 64: of a row, of this launch's value columns per block, of kr
    int max_pages, page_size, n_seqs, nh, window, gate_ld, n_tiles, parts;
    float scale_log2;
    const int *positions, *q_start, *start_pos, *slots, *block_table;
    const float* sink;
    const bf16* gates;
};

__device__ __forceinline__ bool lt_wait(uint32_t mbar, uint32_t parity, volatile int* dead) {
    for (uint32_t i = 0; i < TC_WAIT_LIMIT; ++i) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.b32 %0, 1, 0, p;\n\t}\n" : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
        if (done) return true;
        if (i > 256) {
            if ((i & 63) == 0 && *dead) return false;
            __nanosleep(32);
        }
    }
    *dead = 1;
    return false;
}

__global__ void __launch_bounds__(LT_THREADS, 1)
latent_attention_tc_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map,
                           bf16* __restrict__ out, const LatentTc p, int* status) {
    extern __shared__ unsigned char lt_raw[];
    __shared__ __align__(8) unsigned long long s_q, s_full[2], s_score, s_sum, s_p;     // [0]: key-only blocks, [1]: values
    __shared__ uint32_t s_tmem;
    __shared__ int s_dead, s_req, s_tile, s_issued[2][LT_COPIERS];
    const uint32_t base = (tc_smem(lt_raw) + 1023u) & ~1023u;
    const uint32_t sQ = base, sK = base + p.kb * LT_Q_BLK;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    volatile int* dead = &s_dead;
    ST_PDL_WAIT();
    if (tid == 0) {
        // the last tiles of a request have the longest key ranges: first, all value columns of a tile side by side
        int tile = p.n_tiles - 1 - blockIdx.x / p.parts, req = -1;
        for (int i = 0; i < p.n_seqs; ++i) {
            const int tiles = ((p.q_start[i + 1] - p.q_start[i]) * p.nh + LT_ROWS - 1) / LT_ROWS;
            if (tile < tiles) { req = i; break; }
            tile -= tiles;
        }
        s_req = req;
        s_tile = tile;
        tc_mbar_init(tc_smem(&s_q), LT_COPIERS);
        for (int i = 0; i < 2; ++i) tc_mbar_init(tc_smem(&s_full[i]), LT_COPIERS);
        tc_mbar_init(tc_smem(&s_score), 1);
        tc_mbar_init(tc_smem(&s_sum), 1);
        tc_mbar_init(tc_smem(&s_p), 4);
        tc_mbar_init_fence();
        s_dead = 0;
        for (int i = 0; i < LT_COPIERS; ++i) s_issued[0][i] = s_issued[1][i] = 0;
    }
    __syncthreads();
    const int b = s_req;
    if (b < 0) return;                                        // (the whole block)
    const int tok0 = p.q_start[b], n_rows = (p.q_start[b + 1] - tok0) * p.nh, r0 = s_tile * LT_ROWS;
    if (p.positions[tok0] < 0) return;                        // a padding request of a fixed-shape step
    if (warp == 4 + LT_COPIERS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem(&s_tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    ST_PDL_TRIGGER();                                         // behind the allocation (blocks that have left count as well)
    const uint32_t tmem = s_tmem;                             // O at 0 (64 vb columns), S at 256 and 320, P at 384 and 416
    const int start = p.start_pos[b];
    const int last_row = min(r0 + LT_ROWS, n_rows) - 1;
    const int hi = start + last_row / p.nh + 1;               // keys lo .. hi - 1 are seen by some row of the tile
    const int lo = p.window > 0 ? max(0, start + r0 / p.nh - p.window + 1) : 0;
    const int kt0 = lo / LT_KEYS, n_kt = (hi + LT_KEYS - 1) / LT_KEYS - kt0;
    const int v0 = blockIdx.x % p.parts * p.vb, nv = min(p.vb, p.vb_all - v0);      // this block's values: blocks v0 .. v0 + nv - 1

    if (warp >= 4 && warp < 4 + LT_COPIERS) {
        // ---- copies.  A page without a key this query tile may see may have been given back: its rows (masked, and zeroed as
        // values) are filled from the tile's first live page.
        const int me = warp - 4, n_pg = LT_KEYS / p.page_size;
        const int* bt = p.block_table + (size_t)p.slots[b] * p.max_pages;
        const uint32_t page_bytes = (uint32_t)p.page_size * 128u;
        if (lane == 0) {
            const uint32_t mb = tc_smem(&s_q);
            int mine = 0;
            for (int k = me; k < p.kb; k += LT_COPIERS) ++mine;
            tc_mbar_expect_tx(mb, mine * LT_Q_BLK);
            for (int k = me; k < p.kb; k += LT_COPIERS) tc_tma_load_2d(sQ + k * LT_Q_BLK, &q_map, k * 64, tok0 * p.nh + r0, mb);
            // this warp's pages of a tile: me, and me + 4 where a tile has eight
            auto page_of = [&](int i, int j) -> int {
                if (j >= n_pg || i >= n_kt) return 0;
                const int k0 = (kt0 + i) * LT_KEYS;
                const int first = max(k0, lo) / p.page_size, last = (min(k0 + LT_KEYS, hi) - 1) / p.page_size;
                return bt[min(max(k0 / p.page_size + j, first), last)];
            };
            const int n_mine = (n_pg - me + LT_COPIERS - 1) / LT_COPIERS;        // 0, 1 or 2
            int page[2] = {page_of(0, me), page_of(0, me + LT_COPIERS)};
            bool ok = true;
            for (int i = 0; i < n_kt && ok; ++i) {
                const int next[2] = {page_of(i + 1, me), page_of(i + 1, me + LT_COPIERS)};
                if (((n_mine > 0 && page[0] < 0) || (n_mine > 1 && page[1] < 0)) && status) *status = 1;    // a hole: its rows read as zeros
                for (int part = 0; part < 2; ++part) {
                    // the key-only blocks are free when the scores of the tile before are complete, the values when their
                    // product is
                    if (i > 0) ok = lt_wait(part ? tc_smem(&s_sum) : tc_smem(&s_score), (i - 1) & 1, dead);
                    if (!ok) break;
                    const uint32_t mb = tc_smem(&s_full[part]);
                    tc_mbar_expect_tx(mb, (part ? nv : p.kb - nv) * n_mine * page_bytes);
                    s_issued[part][me] = i + 1;
                    for (int j = 0; j < n_mine; ++j)
                        for (int k = 0; k < p.kb; ++k)
                            if ((k >= v0 && k < v0 + nv) == (part != 0))
                                tc_tma_load_3d(sK + k * LT_K_BLK + (me + LT_COPIERS * j) * page_bytes, &k_map, k * 64, 0, page[j], mb);
                }
                page[0] = next[0];
                page[1] = next[1];
            }
        }
        __syncwarp();
    } else if (warp == 4 + LT_COPIERS && lane == 0) {
        // ---- products
        const uint32_t idesc_s = tc_idesc(LT_ROWS, LT_KEYS, 0, 0), idesc_o = tc_idesc(LT_ROWS, 64 * nv, 0, 1);
        const uint64_t dq = tc_desc(sQ, 16, 1024), dk = tc_desc(sK, 16, 1024);
        const uint64_t dv = tc_desc(sK + v0 * LT_K_BLK, LT_K_BLK, 1024);
        auto scores = [&](int i) -> bool {                    // S of tile i into its buffer
            bool first = true;
            for (int part = 0; part < 2; ++part) {
                if (part == 0 && p.kb == nv) continue;        // every block is a value block
                if (!lt_wait(tc_smem(&s_full[part]), i & 1, dead)) return false;
                tc_fence_after_sync();
                for (int k = 0; k < p.kb; ++k) {
                    if ((k >= v0 && k < v0 + nv) != (part != 0)) continue;
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        tc_mma(tmem + 256 + 64 * (i & 1), dq + ((k * LT_Q_BLK + kk * 32) >> 4), dk + ((k * LT_K_BLK + kk * 32) >> 4),
                               idesc_s, !first);
                        first = false;
                    }
                }
            }
            tc_commit(tc_smem(&s_score));
            return true;
        };
        bool ok = lt_wait(tc_smem(&s_q), 0, dead) && scores(0);
        for (int i = 0; i < n_kt && ok; ++i) {
            ok = lt_wait(tc_smem(&s_p), i & 1, dead);         // P(i) is written (and S(i) read)
            if (!ok) break;
            tc_fence_after_sync();
#pragma unroll
            for (int j = 0; j < LT_KEYS / 16; ++j)
                tc_mma_ts(tmem, tmem + 384 + 32 * (i & 1) + j * 8, dv + ((j * 2048) >> 4), idesc_o, i > 0 || j > 0);
            tc_commit(tc_smem(&s_sum));
            if (i + 1 < n_kt) ok = scores(i + 1);
        }
    } else if (warp < 4) {
        // ---- softmax: thread tid is row tid of the tile and lane tid of tensor memory
        const int row = r0 + tid, tok = row / p.nh;
        const bool live = row < n_rows;
        const int pos = live ? start + tok : -1, first_key = p.window > 0 ? pos - p.window + 1 : 0;
        const uint32_t t_row = tmem + ((uint32_t)(warp * 32) << 16);
        float m_ref = -INFINITY, l_run = 0.f;
        bool ok = true;                                       // the same in every lane of a warp
        for (int i = 0; i < n_kt && ok; ++i) {
            ok = __all_sync(0xffffffffu, lt_wait(tc_smem(&s_score), i & 1, dead));
            if (!ok) break;
            tc_fence_after_sync();
            float s[LT_KEYS];
            tc_ld32(t_row + 256 + 64 * (i & 1), s);
            tc_ld32(t_row + 256 + 64 * (i & 1) + 32, s + 32);
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
                ok = __all_sync(0xffffffffu, lt_wait(tc_smem(&s_sum), (i - 1) & 1, dead));
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
                lt_wait(tc_smem(&s_full[1]), i & 1, dead);
                const int head = min(max(lo - k0, 0), LT_KEYS), tail = max(min(hi - k0, LT_KEYS), head);
                if (lane < nv * 8) {                          // a lane per 16 bytes of a row's values (nv <= 4), a warp per row
                    const uint32_t at = sK + (v0 + lane / 8) * LT_K_BLK + lane % 8 * 16;
                    for (int key = warp; key < LT_KEYS; key += 4)
                        if (key < head || key >= tail)
                            asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};\n" ::"r"(at + key * 128), "r"(0) : "memory");
                }
                tc_fence_async_smem();
            }
            tc_st32(t_row + 384 + 32 * (i & 1), reinterpret_cast<const float*>(w));
            l_run += ((rs[0] + rs[1]) + (rs[2] + rs[3])) + ((rs[4] + rs[5]) + (rs[6] + rs[7]));
            tc_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc_smem(&s_p)) : "memory");
        }
        if (ok) ok = __all_sync(0xffffffffu, lt_wait(tc_smem(&s_sum), (n_kt - 1) & 1, dead));
        tc_fence_after_sync();
        const int h = row % p.nh;
        float k = 0.f;
        if (live) {
            const float snk = p.sink ? p.sink[h] * 1.4426950408889634f : -INFINITY;
            const float mf = fmaxf(m_ref, snk);
            const float c = m_ref == -INFINITY ? 0.f : exp2f(m_ref - mf);
            const float den = l_run * c + (snk > -INFINITY ? exp2f(snk - mf) : 0.f);
            float gate = 1.f;
            if (p.gates) gate = 1.f / (1.f + expf(-load1_cg(p.gates + (size_t)(tok0 + tok) * p.gate_ld + h)));
            k = den > 0.f ? c * gate / den : 0.f;
        }
        if (ok) {
            bf16* dst = out + ((size_t)tok0 * p.nh + row) * (64 * p.vb_all) + 64 * v0;
            for (int c = 0; c < 2 * nv; ++c) {
                float o[32];
                tc_ld32(t_row + c * 32, o);
                tc_ld_wait();
                if (live) {
#pragma unroll
                    for (int e = 0; e < 32; e += 8) {
                        uint4 u;
                        uint32_t* w4 = reinterpret_cast<uint32_t*>(&u);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const __nv_bfloat162 pk = __floats2bfloat162_rn(o[e + 2 * j] * k, o[e + 2 * j + 1] * k);
                            w4[j] = *reinterpret_cast<const uint32_t*>(&pk);
                        }
                        *reinterpret_cast<uint4*>(dst + c * 32 + e) = u;
                    }
                }
                __syncwarp();                                 // the next tcgen05.ld is the whole warp's
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (s_dead && tid == 0) {
        if (status) atomicExch(status, 6);
        tc_wait(tc_smem(&s_q), 0);
        for (int part = 0; part < 2; ++part) {
            int all = s_issued[part][0];
            for (int i = 1; i < LT_COPIERS; ++i) all = min(all, s_issued[part][i]);
            if (all) tc_wait(tc_smem(&s_full[part]), (all - 1) & 1);
        }
        for (int i = 0; i < 20000; ++i) __nanosleep(100);     // and by time the products, and a tile's copies that not all warps began
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
    const unsigned long long kdim[3] = {(unsigned long long)kd, (unsigned long long)page_size, (unsigned long long)n_pages};
    const unsigned long long kst[2] = {(unsigned long long)kd * 2, (unsigned long long)page_stride * 2};
    const unsigned kb[3] = {64, (unsigned)page_size, 1};
    CUtensorMap q_map, k_map;
    if (st_tma_encode_bf16(&q_map, q_lat, 2, qd, qb) ||
        st_tma_encode_bf16_strided(&k_map, (const bf16*)pool + entry_offset, 3, kdim, kst, kb)) return ST_ERR_BAD_ARG;
    LatentTc p;
    p.kb = kd / 64; p.vb_all = kr / 64;
    const int parts = p.parts = (p.vb_all + 3) / 4;
    p.vb = (p.vb_all + parts - 1) / parts;
    p.max_pages = max_pages; p.page_size = page_size; p.n_seqs = n_seqs; p.nh = nh; p.window = window; p.gate_ld = gate_ld;
    p.n_tiles = (int)tiles; p.scale_log2 = scale * 1.4426950408889634f;
    p.positions = positions; p.q_start = q_start; p.start_pos = start_pos; p.slots = slots; p.block_table = block_table;
    p.sink = sink; p.gates = (const bf16*)gates;
    const size_t smem = (size_t)p.kb * (LT_Q_BLK + LT_K_BLK) + 1024;
    const cudaError_t e = cudaFuncSetAttribute(latent_attention_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    return st_launch_pdl("latent_tc", latent_attention_tc_kernel, dim3((unsigned)(tiles * parts)), dim3(LT_THREADS), smem,
                         (cudaStream_t)stream, q_map, k_map, (bf16*)out, p, status);
}
