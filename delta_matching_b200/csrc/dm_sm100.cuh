// Device-side building blocks for the sm_100a kernels: mbarrier, TMA (tiled bulk tensor copies), tensor memory (TMEM)
// allocation and access, tcgen05 MMA issue/commit, shared-memory and instruction descriptors, and bounded waits.
//
// Conventions used by every kernel in this directory:
//  * operand tiles live in shared memory as rows of 128 bytes with the 128-byte swizzle (16-byte chunk index XOR
//    row index mod 8); every tile base is 1024-byte aligned.  The same tile can be consumed K-major (the 128 bytes of a
//    row are the reduction dimension) or MN-major (the 128 bytes of a row are the M or N dimension, rows are the
//    reduction dimension), selected by the descriptor.
//  * every wait on an mbarrier is bounded: after DM_WAIT_LIMIT polls the waiter raises a CTA-wide abort flag, records
//    a status word in global memory and returns; later waits in the same CTA return at once, so the kernel always
//    runs to its end, frees its tensor memory and exits.  Nothing here traps or spins without a limit.
#pragma once
#include <cuda_runtime.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <stdint.h>

#include "dm_launch.cuh"

namespace dm {

#ifndef DM_WAIT_LIMIT
#define DM_WAIT_LIMIT (1u << 22)
#endif

enum : int { DM_DEV_OK = 0, DM_DEV_TIMEOUT = 1 };

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// Byte offset inside a 128-byte-row swizzled tile for (row, byte column).
__device__ __host__ __forceinline__ uint32_t sw128(uint32_t row, uint32_t col_byte) {
    return row * 128u + ((((col_byte >> 4) ^ (row & 7u)) << 4) | (col_byte & 15u));
}

// ---------------------------------------------------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Per-CTA abort state: [0] = abort flag in shared memory, status = global status word (may be null).
struct WaitCtx {
    volatile int* abort_flag;   // shared memory
    int* status;                // global memory, one word per device (dm_device_status reads and clears it)
};
// One look at the barrier without suspending.  On a phase that has already completed this answers in about 60 clocks
// where try_wait takes about 160, so every wait starts with it.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_limit(uint64_t* bar, uint32_t parity, const WaitCtx& ctx, uint32_t limit) {
    if (mbar_test(bar, parity)) return true;
    for (uint32_t it = 0; it < limit; ++it) {
        if (mbar_try(bar, parity)) return true;
        if ((it & 63u) == 63u && *ctx.abort_flag) return false;
    }
    *ctx.abort_flag = 1;
    if (ctx.status) atomicExch(ctx.status, (int)DM_DEV_TIMEOUT);
    return false;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const WaitCtx& ctx) {
    return mbar_wait_limit(bar, parity, ctx, DM_WAIT_LIMIT);
}

// One lane of a converged warp (always the same one).  Under this predicate the compiler knows that a single lane executes the
// asynchronous instruction and feeds its descriptors from uniform registers; under `lane == 0` it cannot, and every
// tcgen05.mma costs the issuing warp more.  Pass 1: 1268 -> 1211 us (B4 N4096 H32 Hk8 causal), 1638 -> 1418 us at head_dim 256
// (B2 N4096 H16 Hk4 full); pass 2: 236 -> 225 us.  Pass 0's role kernel, whose issuing warps wait most of their time, did not gain and
// keeps `lane == 0`.  A warp index taken through __shfl_sync tells the compiler the same about the role branch (pass 2: 225 -> 217 us,
// forward at head_dim 256: 714 -> 699 us).
__device__ __forceinline__ bool elect_one() {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok));
    return ok != 0;
}

// Warp-level arrive: every lane has finished its part (the caller fences as needed), lane 0 arrives once for the warp.
__device__ __forceinline__ void mbar_arrive_warp(uint64_t* bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}
// Named barrier among the first `nthreads` threads of the CTA (id 1..15; id 0 is __syncthreads).
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
// The producer side of a named barrier: counts this warp's threads in and goes on.  `nthreads` is the total of arriving
// and synchronising threads; the arriving side must not get a whole round ahead of the synchronising side.
__device__ __forceinline__ void named_bar_arrive(int id, int nthreads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// Four fp32 additions at one 16-byte address, performed in L2 (rounded to nearest); nothing is returned.
__device__ __forceinline__ void red_add_f32x4(void* to, const float4& y) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(to), "f"(y.x), "f"(y.y), "f"(y.z), "f"(y.w) : "memory");
}

// Register re-allocation between warpgroups (all 128 threads of a warpgroup execute it): the issuer warpgroup gives
// registers back, the compute warpgroups take them.  Counts are multiples of 8.
template <int N> __device__ __forceinline__ void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }

// ---------------------------------------------------------------------------------------------------------- fences
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---------------------------------------------------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// 2-D tiled load global -> shared (this CTA), completion on an mbarrier.  x = byte column (multiple of 16), y = row.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* m, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}
// 2-D tiled store shared -> global.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, int x, int y, const void* smem_src) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                 ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(smem_src)), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_all0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ---------------------------------------------------------------------------------------------------------- TMEM
// Executed by one full warp.  ncols: power of two in [32, 512].
__device__ __forceinline__ void tmem_alloc(uint32_t* holder_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder_smem)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 32 lanes x 32 bit, N consecutive columns: thread t of the warp receives lane (lane_base + t), columns c .. c+N-1.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
// 16 lanes x 256 bit x 4 (32 columns), the matrix-fragment layout: with lane base L (a multiple of 16 inside the warp's quarter),
// register 4 j + 2 a + e of thread t is lane L + t / 4 + 8 a, column c + 8 j + 2 (t % 4) + e.
__device__ __forceinline__ void tmem_ld16x256_x4(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
// The same x 2 (16 columns): register 4 j + 2 a + e, j = 0, 1.
__device__ __forceinline__ void tmem_ld16x256_x2(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
// Four 16 x 8 byte matrices from that layout (register j = the four bytes of fragment j, in register order), stored transposed:
// column i of matrix j becomes 16 consecutive bytes at the address that lane 8 j + i gives.
__device__ __forceinline__ void stmatrix_t_b8_x4(uint32_t saddr, const uint32_t* r) {
    asm volatile("stmatrix.sync.aligned.m16n8.x4.trans.shared.b8 [%0], {%1, %2, %3, %4};"
                 ::"r"(saddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
                 : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
// TMEM address: bits 31..16 lane, bits 15..0 column.
__device__ __forceinline__ uint32_t tmem_addr(uint32_t base, uint32_t lane, uint32_t col) { return base + (lane << 16) + col; }

// ---------------------------------------------------------------------------------------------------------- MMA
// Shared-memory matrix descriptor for a 128-byte-swizzled tile of 128-byte rows (8-row groups 1024 bytes apart).
// K-major: rows are M/N, the 128 bytes of a row are K; one instruction consumes 32 bytes of K, so step k adds 32*k
//          bytes to the start address.
// MN-major: the 128 bytes of a row are M/N (one 128-wide atom), rows are K; one instruction consumes 32 rows = 4096
//          bytes, so step k adds 4096*k bytes.  The leading byte offset (distance between 128-wide atoms along M/N) is
//          unused with a single atom.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);        // start address, 16-byte units
    d |= (uint64_t)1 << 16;                          // leading byte offset (16-byte units); unused here
    d |= (uint64_t)(1024u >> 4) << 32;               // stride byte offset: 8-row group pitch
    d |= (uint64_t)1 << 46;                          // descriptor version for sm_100
    d |= (uint64_t)2 << 61;                          // layout type: 128-byte swizzle
    return d;
}
// The same descriptor as two 32-bit words: only the low word depends on the address, so an issuing thread keeps one
// register per buffer and advances it by (bytes >> 4); the high word is a constant.
constexpr uint32_t kDescHiSw128 = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t smem_desc_lo_sw128(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | (1u << 16); }

// Instruction descriptor, kind::f8f6f4, e4m3 x e4m3 -> fp32, dense.
__host__ __device__ constexpr uint32_t idesc_e4m3(int M, int N, bool a_mn_major, bool b_mn_major) {
    return (1u << 4)                               // D format fp32
           | (0u << 7) | (0u << 10)                // A, B format e4m3
           | ((a_mn_major ? 1u : 0u) << 15) | ((b_mn_major ? 1u : 0u) << 16)
           | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// D[tmem] (+)= A[smem] * B[smem]; issued by ONE thread.
__device__ __forceinline__ void umma_e4m3(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The same with descriptors given by their low words (high word = kDescHiSw128) and a compile-time accumulate flag.
template <bool kAccumulate>
__device__ __forceinline__ void umma_e4m3_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 da, {%1, %5};\n\t"
        "mov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], da, db, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "n"(kAccumulate ? 1 : 0), "n"(kDescHiSw128)
        : "memory");
}
__device__ __forceinline__ void umma_e4m3_lo_rt(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 da, {%1, %5};\n\t"
        "mov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], da, db, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(kDescHiSw128)
        : "memory");
}
// The A operand read from tensor memory instead of shared memory (always K-major): lane = row of A (M = 128), each 32-bit
// column holds four consecutive e4m3 elements of K (lowest byte first), so one K step of 32 is 8 columns and step k reads
// columns [a_tmem + 8 k, a_tmem + 8 k + 8).  B comes from shared memory as above.
template <bool kAccumulate>
__device__ __forceinline__ void umma_e4m3_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], [%1], db, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(idesc), "n"(kAccumulate ? 1 : 0), "n"(kDescHiSw128)
        : "memory");
}
// Arrive on an mbarrier once every MMA issued so far by this thread has completed (implies fence::before_thread_sync).
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// ---------------------------------------------------------------------------------------------------------- math
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Packed fp32 pairs (one instruction for two lanes of arithmetic, IEEE round-to-nearest per component, so the results
// carry the bits of the scalar operations): y = x * m + c, y = x * m, on two values at a time.
__device__ __forceinline__ void fma2(float& y0, float& y1, float x0, float x1, float m, float c0, float c1) {
    const float2 r = __ffma2_rn(make_float2(x0, x1), make_float2(m, m), make_float2(c0, c1));
    y0 = r.x;
    y1 = r.y;
}
__device__ __forceinline__ void mul2(float& y0, float& y1, float x0, float x1, float m0, float m1) {
    const float2 r = __fmul2_rn(make_float2(x0, x1), make_float2(m0, m1));
    y0 = r.x;
    y1 = r.y;
}
__device__ __forceinline__ void add2(float& y0, float& y1, float x0, float x1) {
    const float2 r = __fadd2_rn(make_float2(y0, y1), make_float2(x0, x1));
    y0 = r.x;
    y1 = r.y;
}
// max of three in one instruction
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// max(|a|, |b|, |c|)
__device__ __forceinline__ float fmax3_abs(float a, float b, float c) {
    float d;
    asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// Four fp32 -> four e4m3 (round-to-nearest-even, saturate-to-finite), the first in bits 0..7.  Joined by a 16-bit pair move, which the
// second conversion does on the way (an `or` with a shift costs an instruction of its own, one per four codes: forward at B4 N4096 H32
// causal 504 -> 502 us).
__device__ __forceinline__ uint32_t cvt_e4m3x4(float a, float b, float c, float d) {
    uint32_t r;
    asm("{\n\t.reg .b16 l, h;\n\t"
        "cvt.rn.satfinite.e4m3x2.f32 l, %2, %1;\n\t"
        "cvt.rn.satfinite.e4m3x2.f32 h, %4, %3;\n\t"
        "mov.b32 %0, {l, h};\n\t}"
        : "=r"(r)
        : "f"(a), "f"(b), "f"(c), "f"(d));
    return r;
}

}  // namespace dm
