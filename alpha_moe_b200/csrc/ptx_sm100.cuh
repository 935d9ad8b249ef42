// Thin inline-PTX wrappers for sm_100a: mbarrier, TMA (cp.async.bulk.tensor), cp.async,
// tcgen05 (TMEM alloc, UMMA issue/commit, TMEM loads) and bf16x2 global reductions.
//
// This header takes the place of the reference's Hopper helper layer
// (csrc/kernels/fused_moe_w8a8/fused_moe_w8a8_up_down_acc.cu:41-633: wgmma wrappers,
// Hopper smem descriptors, TMA/mbarrier helpers, stmatrix); none of that layer can be
// assembled for sm_100a, so everything here is written against the Blackwell
// instructions instead.  Every wait is bounded: a wait that runs out records a status
// word and returns false, it never spins forever.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace amoe {

// ---------------------------------------------------------------------------------------------
// status word written by a kernel whose bounded wait ran out (0 = healthy)
struct KernelStatus {
    int code;     // 0 ok, otherwise WAIT_* below
    int block;    // blockIdx.x of the first CTA that gave up
    int where;    // role-specific tag (which barrier)
    int iter;     // pipeline iteration
};
enum : int { ST_OK = 0, ST_WAIT_TIMEOUT = 1, ST_SMEM_MISALIGNED = 2 };

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// --------------------------------------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Arrival without release ordering: for hand-offs where the arriving thread has written nothing the
// waiter will read (e.g. "TMEM has been read", "ring slot is free").  A default (release) arrive would
// also wait for this thread's outstanding global reductions to be acknowledged by L2.
__device__ __forceinline__ void mbar_arrive_relaxed(uint64_t* bar) {
    asm volatile("mbarrier.arrive.relaxed.cta.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_relaxed_n(uint64_t* bar, uint32_t n) {
    asm volatile("mbarrier.arrive.relaxed.cta.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(n) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
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

// Limit of one wait, in SM clock cycles (about a second at B200 clocks).
constexpr long long kWaitLimitCycles = 2000000000LL;

// First wait of a launch to run out: raises the CTA's abort flag and records where it was.
__device__ __forceinline__ void record_run_out(volatile int* abort_flag, KernelStatus* status, int where, int iter) {
    *abort_flag = 1;
    if (atomicCAS(&status->code, ST_OK, ST_WAIT_TIMEOUT) == ST_OK) {
        status->block = blockIdx.x;
        status->where = where;
        status->iter = iter;
    }
}

// Bounded wait.  `abort_flag` is a CTA-shared word: once any thread of the CTA gives up, every
// other waiter of that CTA returns false at its next poll, so the CTA unwinds as a whole.
// (Kept inline: a device function call inside a role that has resized its register allotment with
// setmaxnreg does not get through register allocation.)
// Each thread decides for itself: for a single lane, or for threads that need no other lane afterwards.
__device__ __forceinline__ bool mbar_wait_limit(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                KernelStatus* status, int where, int iter, long long limit_cycles) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 32; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > limit_cycles) {
            record_run_out(abort_flag, status, where, iter);
            return false;
        }
    }
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          KernelStatus* status, int where, int iter) {
    return mbar_wait_limit(bar, parity, abort_flag, status, where, iter, kWaitLimitCycles);
}

// The same for a whole warp whose next steps need all 32 lanes (elect.sync, __syncwarp): the lanes vote on every poll, so
// all of them get the same answer by construction.  With a decision per lane, one that gives up (the abort flag, its own
// clock) while another has seen the barrier complete would leave the other at the next full-mask instruction for good.
__device__ __forceinline__ bool mbar_wait_warp_limit(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                     KernelStatus* status, int where, int iter, long long limit_cycles) {
    if (__all_sync(0xFFFFFFFFu, mbar_try_wait(bar, parity))) return true;
    const long long t0 = clock64();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 32; ++i)
            if (__all_sync(0xFFFFFFFFu, mbar_try_wait(bar, parity))) return true;
        const bool run_out = clock64() - t0 > limit_cycles;
        if (run_out) record_run_out(abort_flag, status, where, iter);
        if (__any_sync(0xFFFFFFFFu, run_out || *abort_flag != 0)) return false;
    }
}
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                               KernelStatus* status, int where, int iter) {
    return mbar_wait_warp_limit(bar, parity, abort_flag, status, where, iter, kWaitLimitCycles);
}
// The last wait of a CTA that gives up: first phase of either of two mbarriers, or `limit_cycles`, whatever the abort flag says.
__device__ __forceinline__ bool mbar_wait_either_limit(uint64_t* a, uint64_t* b, long long limit_cycles) {
    const long long t0 = clock64();
    for (;;) {
        if (mbar_try_wait(a, 0) || mbar_try_wait(b, 0)) return true;
        if (clock64() - t0 > limit_cycles) return false;
    }
}
constexpr long long kLandingCycles = 2000000LL;      // about a millisecond: a thousand times what a store to a peer takes
// A whole warp waits until the counter `turn` in shared memory has reached `it`; one answer for all lanes, as above.
__device__ __forceinline__ bool turn_wait_warp_limit(volatile int* turn, int it, volatile int* abort_flag,
                                                     KernelStatus* status, int where, long long limit_cycles) {
    if (__all_sync(0xFFFFFFFFu, *turn >= it)) return true;
    const long long t0 = clock64();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 8; ++i)
            if (__all_sync(0xFFFFFFFFu, *turn >= it)) return true;
        const bool run_out = clock64() - t0 > limit_cycles;
        if (run_out) record_run_out(abort_flag, status, where, it);
        if (__any_sync(0xFFFFFFFFu, run_out || *abort_flag != 0)) return false;
    }
}
__device__ __forceinline__ bool turn_wait_warp(volatile int* turn, int it, volatile int* abort_flag, KernelStatus* status,
                                               int where) {
    return turn_wait_warp_limit(turn, it, abort_flag, status, where, kWaitLimitCycles);
}

// --------------------------------------------------------------------------------------------- clusters / DSMEM
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Hardware barrier over all threads of all CTAs of the cluster (used once, right after barrier set-up,
// where every CTA arrives unconditionally).
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The same without any ordering of memory accesses: at the end of a kernel, where no CTA may go while a peer may still issue writes
// into or reads from its shared memory.  (A releasing arrival would wait for the acknowledgement of all reductions.)  Writes that a
// peer has issued are not waited for: their receiver does that on the mbarrier that counts them.
__device__ __forceinline__ void cluster_sync_all_relaxed() {
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
// shared::cta address -> address of the same location in the shared memory of CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Two floats into a peer's shared memory, counted as 8 bytes by the peer's mbarrier (both addresses from mapa_shared): who has
// waited for that barrier sees them.
__device__ __forceinline__ void st_async_f32x2(uint32_t cluster_addr, float a, float b, uint32_t cluster_bar) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(__float_as_uint(a)), "r"(__float_as_uint(b)));
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];"
                 ::"r"(cluster_addr), "l"(v), "r"(cluster_bar) : "memory");
}
__device__ __forceinline__ float ld_dsmem_f32(uint32_t cluster_addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr) : "memory");
    return v;
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait on a barrier that CTAs of the cluster arrive on (acquire at cluster scope).
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                  KernelStatus* status, int where, int iter) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 32; ++i)
            if (mbar_try_wait_cluster(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > kWaitLimitCycles) {
            record_run_out(abort_flag, status, where, iter);
            return false;
        }
    }
}

// --------------------------------------------------------------------------------------------- proxies
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// --------------------------------------------------------------------------------------------- TMA
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* m) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}

// --------------------------------------------------------------------------------------------- cp.async (16 B)
// src_bytes = 16 copies, src_bytes = 0 writes 16 zero bytes (src must still be a valid address).
__device__ __forceinline__ void cp_async_16(uint32_t dst_smem, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst_smem), "l"(src), "r"(src_bytes) : "memory");
}
// The mbarrier receives one arrival from this thread once all cp.async copies it has issued so far have
// landed (asynchronously: the thread does not wait).  .noinc: the arrival is part of the barrier's
// expected count, so a phase cannot complete before every gathering thread's copies are in.
__device__ __forceinline__ void cp_async_mbar_arrive_noinc(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_n(uint64_t* bar, uint32_t n) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// --------------------------------------------------------------------------------------------- tcgen05 / TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor, K-major operand stored as rows of 128 bytes with the 128-byte
// swizzle (what TMA writes with CU_TENSOR_MAP_SWIZZLE_128B); the leading offset is unused for this
// layout, descriptor version 1, layout type 2.
// `sbo` is the distance between consecutive 8-row groups of the operand: 1024 for a dense tile, 2048
// to take every other 8-row group of a tile (how the gate / up halves of the interleaved `w` rows are
// picked apart without moving any data).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr, uint32_t sbo = 1024u) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);        // start address  [0,14)
    d |= static_cast<uint64_t>(sbo >> 4) << 32;                     // stride byte offset [32,46)
    d |= static_cast<uint64_t>(1) << 46;                            // version [46,48)
    d |= static_cast<uint64_t>(2) << 61;                            // SWIZZLE_128B [61,64)
    return d;
}
// Instruction descriptor for kind::f8f6f4, e4m3 x e4m3 -> f32, both operands K-major.
__host__ __device__ constexpr uint32_t umma_idesc_e4m3(uint32_t m, uint32_t n) {
    return (1u << 4) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
// One 128-deep K chunk (four K=32 steps) of two independent accumulators:
//   D0 = A0 * B0, D1 = A1 * B1   (fresh accumulation: the first step overwrites D).
// All eight instructions sit in one asm block so that the issuing thread spends no instructions
// between them; descriptors advance by 32 bytes (2 in units of 16 B) per K step.
__device__ __forceinline__ void umma_f8_chunk2(uint32_t d0, uint32_t d1, uint64_t a0, uint64_t a1, uint64_t b0,
                                               uint64_t b1, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred pf, pt;\n\t.reg .b64 a0k, a1k, b0k, b1k;\n\t"
        "setp.ne.b32 pf, 0, 0;\n\tsetp.eq.b32 pt, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %2, %4, %6, pf;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%1], %3, %5, %6, pf;\n\t"
        "add.u64 a0k, %2, 2;\n\tadd.u64 a1k, %3, 2;\n\tadd.u64 b0k, %4, 2;\n\tadd.u64 b1k, %5, 2;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a0k, b0k, %6, pt;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%1], a1k, b1k, %6, pt;\n\t"
        "add.u64 a0k, %2, 4;\n\tadd.u64 a1k, %3, 4;\n\tadd.u64 b0k, %4, 4;\n\tadd.u64 b1k, %5, 4;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a0k, b0k, %6, pt;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%1], a1k, b1k, %6, pt;\n\t"
        "add.u64 a0k, %2, 6;\n\tadd.u64 a1k, %3, 6;\n\tadd.u64 b0k, %4, 6;\n\tadd.u64 b1k, %5, 6;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a0k, b0k, %6, pt;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%1], a1k, b1k, %6, pt;\n\t}"
        ::"r"(d0), "r"(d1), "l"(a0), "l"(a1), "l"(b0), "l"(b1), "r"(idesc)
        : "memory");
}
// Same for a single accumulator.
__device__ __forceinline__ void umma_f8_chunk1(uint32_t d0, uint64_t a0, uint64_t b, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred pf, pt;\n\t.reg .b64 a0k, bk;\n\t"
        "setp.ne.b32 pf, 0, 0;\n\tsetp.eq.b32 pt, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, pf;\n\t"
        "add.u64 a0k, %1, 2;\n\tadd.u64 bk, %2, 2;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a0k, bk, %3, pt;\n\t"
        "add.u64 a0k, %1, 4;\n\tadd.u64 bk, %2, 4;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a0k, bk, %3, pt;\n\t"
        "add.u64 a0k, %1, 6;\n\tadd.u64 bk, %2, 6;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a0k, bk, %3, pt;\n\t}"
        ::"r"(d0), "l"(a0), "l"(b), "r"(idesc)
        : "memory");
}
// D[tmem] (+)= A[smem] * B[smem]; issued by one thread.
__device__ __forceinline__ void umma_f8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// One lane of a converged warp.  tcgen05.mma takes its descriptors from uniform registers: inside `if (lane == 0)`, which
// the compiler has to treat as divergent, its operands have to be made uniform first; with a warp-uniform loop around an
// elected lane they are uniform to begin with.
__device__ __forceinline__ bool elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}
// mbarrier arrives once all UMMAs issued so far by this thread have completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
// 32 lanes x 16 consecutive 32-bit columns: thread t of the warp gets lane (lane_base + t).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Two accumulators' 32 lanes x 16 columns as fragments (two 16-lane loads each): v[h][4i], v[h][4i + 1] of thread t = lane
// 16h + t / 4, columns 8i + 2 (t % 4) and the next; v[h][4i + 2], v[h][4i + 3] = the same columns of lane 16h + 8 + t / 4.
// One asm block with the wait, so that the results are plain outputs and no use of them comes before it: a wait of its own that
// took them as in-and-out operands made the compiler move registers (DeepSeek-V3 TP8 shard, operator, calls in a row, M = 777
// 255.3 -> 252.6 us, M = 1024 273 -> 270; part of it from the warp index that is uniform to the compiler).
__device__ __forceinline__ void tmem_ld_two_frag16_wait(uint32_t addr_a, uint32_t addr_b, uint32_t (&a)[2][8], uint32_t (&b)[2][8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%32];\n\t"
        "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%33];\n\t"
        "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%16, %17, %18, %19, %20, %21, %22, %23}, [%34];\n\t"
        "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%24, %25, %26, %27, %28, %29, %30, %31}, [%35];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=&r"(a[0][0]), "=&r"(a[0][1]), "=&r"(a[0][2]), "=&r"(a[0][3]), "=&r"(a[0][4]), "=&r"(a[0][5]), "=&r"(a[0][6]), "=&r"(a[0][7]),
          "=&r"(a[1][0]), "=&r"(a[1][1]), "=&r"(a[1][2]), "=&r"(a[1][3]), "=&r"(a[1][4]), "=&r"(a[1][5]), "=&r"(a[1][6]), "=&r"(a[1][7]),
          "=&r"(b[0][0]), "=&r"(b[0][1]), "=&r"(b[0][2]), "=&r"(b[0][3]), "=&r"(b[0][4]), "=&r"(b[0][5]), "=&r"(b[0][6]), "=&r"(b[0][7]),
          "=&r"(b[1][0]), "=&r"(b[1][1]), "=&r"(b[1][2]), "=&r"(b[1][3]), "=&r"(b[1][4]), "=&r"(b[1][5]), "=&r"(b[1][6]), "=&r"(b[1][7])
        : "r"(addr_a), "r"(addr_a + (16u << 16)), "r"(addr_b), "r"(addr_b + (16u << 16))
        : "memory");
}
// Four 8 x 8 matrices of 16-bit values, stored transposed: thread t holds (row t / 4, columns 2 (t % 4) and the next)
// of each; thread t's address is that of row t % 8 of transposed matrix t / 8.
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, const uint32_t (&m)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};"
                 ::"r"(addr), "r"(m[0]), "r"(m[1]), "r"(m[2]), "r"(m[3]) : "memory");
}

// --------------------------------------------------------------------------------------------- packed fp32 pairs
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack_u32x2(uint32_t lo, uint32_t hi) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
    return d;
}
__device__ __forceinline__ f32x2 pack_f32x2(float lo, float hi) { return pack_u32x2(__float_as_uint(lo), __float_as_uint(hi)); }
__device__ __forceinline__ void unpack_f32x2(f32x2 d, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(d));
}
__device__ __forceinline__ f32x2 fma_f32x2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 mul_f32x2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// --------------------------------------------------------------------------------------------- misc
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
__device__ __forceinline__ void red_add_bf16x2(__nv_bfloat16* addr, float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    // no "memory" clobber: nothing in a kernel reads `out` back, and the clobber would serialise the
    // shared-memory loads of neighbouring iterations behind each reduction
    asm volatile("red.global.add.noftz.bf16x2 [%0], %1;" ::"l"(addr), "r"(*reinterpret_cast<uint32_t*>(&v)));
}
// Same, issued only where `row < nrows` (no branch: the bound check is a predicate on the instruction).
__device__ __forceinline__ void red_add_bf16x2_if(__nv_bfloat16* addr, float lo, float hi, int row, int nrows) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %2, %3;\n\t"
        "@p red.global.add.noftz.bf16x2 [%0], %1;\n\t}"
        ::"l"(addr), "r"(*reinterpret_cast<uint32_t*>(&v)), "r"(row), "r"(nrows));
}
// 16 bytes = 8 consecutive bf16 values in one reduction, issued only where `pred` holds.
__device__ __forceinline__ void red_add_v4_bf16x2_raw_if(__nv_bfloat16* addr, const uint4& w, bool pred) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "@p red.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};\n\t}"
        ::"l"(addr), "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w), "r"(static_cast<uint32_t>(pred)));
}
// One packed pair, issued only where `pred` holds.
__device__ __forceinline__ void red_add_bf16x2_raw_if(__nv_bfloat16* addr, uint32_t w, bool pred) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t"
        "@p red.global.add.noftz.bf16x2 [%0], %1;\n\t}"
        ::"l"(addr), "r"(w), "r"(static_cast<uint32_t>(pred)));
}
// Register re-balancing between warpgroups (all four warps of a warpgroup must execute it).
template <int N>
__device__ __forceinline__ void setmaxnreg_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void setmaxnreg_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}
// Global load that the compiler keeps where it is written (used to request small schedule words at kernel entry, ahead of the
// set-up work whose latency they then overlap).  Not ld.global.nc or __ldg, which want memory that nothing writes while the
// kernel runs: as a programmatic dependent it is there before the kernel in front has written them.
__device__ __forceinline__ int ld_global_s32(const int* p) {
    int v;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
// Programmatic dependent launch.  A kernel launched with the programmatic-serialisation attribute may start while
// the kernel in front of it in the stream is still running; griddep_wait() returns once that kernel has completed and
// its writes are visible (at once if there is no such dependency), so nothing it produced may be read before.
// griddep_launch_dependents() tells the scheduler that the kernel behind this one may start now.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

}  // namespace amoe
