// Device helpers for kernels on the 5th-generation tensor cores (tcgen05): shared-memory matrix
// descriptors, instruction descriptors, tcgen05.mma / commit / ld / st in inline PTX, bounded mbarrier
// waits, and TMA (cp.async.bulk.tensor) loads that complete on an mbarrier.  Included by the attention
// kernels for portions of prompts; no reference counterpart (the reference's kernels use mma.sync-era
// instructions: src/csrc/kernel/xformers_attention.cu).
#pragma once
#include "common.cuh"

#define TC_BM 128   // query rows of a tile: the lanes of tensor memory
#define TC_BN 64    // keys of a tile
#define TC_LOG2E 1.4426950408889634f
#define TC_WAIT_LIMIT (1u << 21)     // polls of about 50 ns each: a wait gives up after roughly 0.1 s

__device__ __forceinline__ uint32_t tc_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void tc_cp16(uint32_t dst, const void* src, bool pred) {
    const int n = pred ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n));
}
__device__ __forceinline__ void tc_cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void tc_cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }
// writes made through the generic proxy (cp.async, st.shared) become visible to the tensor cores' async proxy
__device__ __forceinline__ void tc_fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

__device__ __forceinline__ float tc_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}

// sm_100 arithmetic on pairs of floats and the three-input maximum: fewer instructions for the softmax threads
__device__ __forceinline__ void tc_fma2(float& d0, float& d1, float a0, float a1, float b, float c) {   // a * b + c
    asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmov.b64 c, {%5, %5};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}\n"
        : "=f"(d0), "=f"(d1) : "f"(a0), "f"(a1), "f"(b), "f"(c));
}
__device__ __forceinline__ void tc_add2(float& d0, float& d1, float a0, float a1) {                      // d += a
    asm("{\n\t.reg .b64 a, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 d, {%0, %1};\n\t"
        "add.rn.f32x2 d, d, a;\n\tmov.b64 {%0, %1}, d;\n\t}\n"
        : "+f"(d0), "+f"(d1) : "f"(a0), "f"(a1));
}
__device__ __forceinline__ float tc_max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// shared-memory matrix descriptor: 128-byte swizzle, descriptor version 1 (sm_100)
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32) | (1ull << 46) | (2ull << 61);
}
// instruction descriptor, kind::f16: bfloat16 operands, float accumulator
__device__ __forceinline__ uint32_t tc_idesc(int m, int n, int a_mn_major, int b_mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn_major << 15) | ((uint32_t)b_mn_major << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, int accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// the same with the A operand in tensor memory (lanes = rows, 8 columns of packed 16-bit pairs per K = 16)
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, int accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
                 ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(mbar) : "memory");
}
// One lane of a converged warp, the same one each time.  A warp that issues products or copies runs its loops as a whole, with the
// waits, and only the issue stands under this: the compiler then knows that addresses and descriptors are the same in all
// lanes and keeps them in uniform registers.  Under `lane == 0` it does not: a product of 128 x 16 x 16 from tensor memory took 46
// clocks to issue with constant offsets, 115 with computed ones, and takes 9 this way; a copy of one box 54 and 16.
__device__ __forceinline__ bool tc_elect() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
    return p != 0;
}
// a thread's warp, known to be the same in all lanes
__device__ __forceinline__ int tc_warp() { return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); }
// bounded wait for the given phase parity; false: gave up
__device__ __forceinline__ bool tc_wait(uint32_t mbar, uint32_t parity) {
    for (uint32_t i = 0; i < TC_WAIT_LIMIT; ++i) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.b32 %0, 1, 0, p;\n\t}\n" : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
        if (done) return true;
        if (i > 64) __nanosleep(32);
    }
    return false;
}
// The same by a whole warp, with one answer for all its lanes, which also ends when the block has been marked dead, and marks it
// when the limit is reached.  try_wait: the hardware holds the warp until the phase completes or a time of about a microsecond
// is over, so that waiting warps take no issue slots from working ones.
#define TC_TRY_LIMIT (1u << 17)       // tries: at least 0.1 s, whatever a try's time is; no warp that others wait for may be busy for long
__device__ __forceinline__ bool tc_wait_warp(uint32_t mbar, uint32_t parity, volatile int* dead) {
    bool ok = false;
    for (uint32_t i = 0; i < TC_TRY_LIMIT; ++i) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
                     "selp.b32 %0, 1, 0, p;\n\t}\n" : "=r"(done) : "r"(mbar), "r"(parity), "r"(1000u) : "memory");
        if (done) { ok = true; break; }
        if (*dead) break;
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) *dead = 1;
    return ok;
}
// 32 consecutive float columns of this thread's TMEM lane: the load is only issued here; the values
// may be used after tc_ld_wait() (several loads can be in flight under one wait)
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float* v) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }

__device__ __forceinline__ void tc_st32(uint32_t taddr, const float* v) {
    const uint32_t* r = reinterpret_cast<const uint32_t*>(v);
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};\n"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                   "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
                   "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]),
                   "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
// barrier of one warpgroup; the ids are immediates: with a register operand the compiler reserves all
// sixteen barriers for the block, and two such blocks do not fit one SM
__device__ __forceinline__ void tc_wg_sync(int wgi) {
    if (wgi == 0) asm volatile("bar.sync 1, 128;\n" ::: "memory");
    else if (wgi == 1) asm volatile("bar.sync 2, 128;\n" ::: "memory");
    else if (wgi == 2) asm volatile("bar.sync 3, 128;\n" ::: "memory");
    else asm volatile("bar.sync 4, 128;\n" ::: "memory");
}

// ---- mbarriers and TMA -----------------------------------------------------------------------------
__device__ __forceinline__ void tc_mbar_init(uint32_t mbar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(mbar), "r"(count) : "memory");
}
__device__ __forceinline__ void tc_mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory"); }
// one arrival that also announces `bytes` of asynchronous copies which will complete on the barrier
__device__ __forceinline__ void tc_mbar_expect_tx(uint32_t mbar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(mbar), "r"(bytes) : "memory");
}
// TMA load of one box of a rank-3 tensor map into shared memory (no multicast).  c0 is the innermost
// coordinate; c0 x element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tc_tma_load_3d(uint32_t dst, const void* tmap, int c0, int c1, int c2, uint32_t mbar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
                 "[%0], [%1, {%2, %3, %4}], [%5];\n"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(c2), "r"(mbar) : "memory");
}
__device__ __forceinline__ void tc_tma_load_2d(uint32_t dst, const void* tmap, int c0, int c1, uint32_t mbar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
                 "[%0], [%1, {%2, %3}], [%4];\n"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(mbar) : "memory");
}
__device__ __forceinline__ void tc_tma_load_4d(uint32_t dst, const void* tmap, int c0, int c1, int c2, int c3, uint32_t mbar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
                 "[%0], [%1, {%2, %3, %4, %5}], [%6];\n"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(mbar) : "memory");
}
