// Thin inline-PTX wrappers for sm_100a: mbarrier, TMA (cp.async.bulk.tensor), tcgen05 (UMMA +
// tensor memory).  Every wait is bounded: after WAIT_LIMIT_CYCLES it reports a code through an
// error word and returns false so the caller can unwind (free TMEM, leave) instead of hanging.
#pragma once
#include <cuda.h>
#include <cstdint>

namespace ptx {

// About one second at B200 clocks; far above any legitimate wait inside these kernels.
constexpr long long WAIT_LIMIT_CYCLES = 2000000000LL;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// ---- mbarrier -------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// generic-proxy writes to shared memory -> visible to the async proxy (TMA / tcgen05.mma reads)
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
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

// Non-blocking look at a phase.  (try_wait may park the thread for a hardware-defined time, about 4 us on B200, before it
// says no: code with something else to do meanwhile must not use it.)
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
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

// Bounded wait.  `abort_flag` lives in shared memory: the first waiter that runs out of time sets it (and the global error
// word) so every other waiter of the CTA leaves at once.  The first look is all that is inlined; what follows a miss is a
// call.  With the retry loop, the clock and the abort flag inlined behind the first look, an MMA step (four 128 x 48 x 16 MMAs,
// one commit) whose barrier was complete already took 294 cycles, like this 136, without any wait 97: the loop's second
// way out makes the compiler guard every wait of a divergent thread with convergence barriers.  CALL = false keeps it all inline, for
// kernels that have no registers to spare around a call.
// mbarrier.try_wait itself parks the thread for a hardware-defined interval (about 8000 cycles), so the loop is cheap; the clock
// and the abort flag are looked at only after the first and every 256th failed try.
template <bool CLUSTER> __device__ __forceinline__ bool mbar_look(uint32_t bar, uint32_t parity) {     // CLUSTER: acquire at cluster scope
    uint32_t ok;
    if (CLUSTER)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// PAIR: whoever gives up sets the abort flag of both CTAs of the cluster (each lies at the same offset) before it returns, so what its
// warp arrives on in the other CTA afterwards cannot pass for a success there.
template <bool PAIR>
__device__ __forceinline__ bool mbar_give_up(volatile uint32_t* abort_flag) {
    if (PAIR) {
        const uint32_t at = smem_u32(const_cast<const uint32_t*>(abort_flag));
        asm volatile(
            "{\n\t.reg .u32 r, a;\n\t"
            "mov.u32 r, %%cluster_ctarank;\n\t"
            "xor.b32 r, r, 1;\n\t"
            "mapa.shared::cluster.u32 a, %0, r;\n\t"
            "st.volatile.shared::cluster.u32 [a], 1;\n\t"
            "fence.acq_rel.cluster;\n\t}"
            ::"r"(at) : "memory");
    }
    return false;
}
template <bool CLUSTER, bool PAIR>
__device__ __forceinline__ bool mbar_keep_looking(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, int* err_word, int code) {
    long long t0 = 0;
    for (uint32_t spin = 1;; ++spin) {
        if (mbar_look<CLUSTER>(bar, parity)) return true;
        if ((spin & 255u) == 0u || spin == 1u) {
            if (*abort_flag) return mbar_give_up<PAIR>(abort_flag);
            const long long now = clock64();
            if (t0 == 0) t0 = now;
            else if (now - t0 > WAIT_LIMIT_CYCLES) {
                *abort_flag = 1u;
                if (err_word) atomicCAS(err_word, 0, code);
                return mbar_give_up<PAIR>(abort_flag);
            }
        }
    }
}
template <bool CLUSTER, bool PAIR>
static __device__ __noinline__ bool mbar_missed(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, int* err_word, int code) {
    return mbar_keep_looking<CLUSTER, PAIR>(bar, parity, abort_flag, err_word, code);
}
template <bool CALL = true, bool PAIR = false, bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag, int* err_word, int code) {
    if (mbar_look<CLUSTER>(smem_u32(bar), parity)) return true;
    return CALL ? mbar_missed<CLUSTER, PAIR>(smem_u32(bar), parity, abort_flag, err_word, code)
                : mbar_keep_looking<CLUSTER, PAIR>(smem_u32(bar), parity, abort_flag, err_word, code);
}
// on a local barrier that the other CTA of a pair arrives on too
template <bool CALL = true, bool PAIR = true>
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag, int* err_word, int code) {
    return mbar_wait<CALL, PAIR, true>(bar, parity, abort_flag, err_word, code);
}

// ---- TMA ------------------------------------------------------------------------------
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* m) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
}
// 2-D tiled load, completes `bytes` on the mbarrier.  x is the innermost (contiguous)
// coordinate in elements and must make x*elemsize a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}

// 1-D bulk copy global -> shared, completes `bytes` on the mbarrier.  Both addresses 16-byte aligned, bytes a
// multiple of 16.
__device__ __forceinline__ void bulk_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// ---- tensor memory + UMMA ---------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {  // whole warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {    // whole warp
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem desc] * B[smem desc]; fp16 operands, fp32 accumulate; one thread issues.
__device__ __forceinline__ void umma_f16_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// mbarrier arrives once every MMA issued so far by this thread has finished
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// ---- CTA pairs (cta_group::2): one MMA spans the tensor cores of two SMs ------------------------------------------
// The two CTAs of a cluster of two hold 128 rows of A each and half of B's rows each; the accumulator of CTA r (rows
// 128 r .. 128 r + 127 of the 256-row result) sits in that CTA's tensor memory.  One thread of the even-ranked CTA issues
// the MMAs; operand descriptors name the same shared-memory offsets in both CTAs.  Per SM the MMA then reads its A rows and
// only half of B from shared memory, which is what takes the shared-memory pipe off the critical path.
__device__ __forceinline__ uint32_t cluster_ctarank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync_all() {   // every thread of every CTA of the cluster
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* dst_smem, uint32_t ncols) {  // one warp of each CTA of the pair
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_pair_f16_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// the barrier at this shared-memory offset in both CTAs of the pair gets one arrival once every MMA issued so far by this
// thread has finished
__device__ __forceinline__ void umma_pair_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
// Arrival on the barrier at this offset in CTA `rank` of the cluster.  Plain form (release at CTA scope), as for a local
// barrier: what the arrival publishes are shared-memory stores that fence.proxy.async has already handed to the async
// proxy, which is the proxy the other CTA's MMA reads them through.  (With .release.cluster the arriving unpack thread
// stalled about a thousand cycles per stage, which made the pair slower than two single CTAs.)
__device__ __forceinline__ void mbar_arrive_cluster(uint64_t* bar, uint32_t rank) {
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_u32(bar)), "r"(rank));
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(ra) : "memory");
}
// 32 lanes x 16 consecutive fp32 columns -> 16 registers per thread (lane i of the warp reads
// TMEM lane (taddr.lane + i)).  Warp w of a CTA may only touch lanes 32*(w%4) .. +31.
__device__ __forceinline__ void tmem_ld_x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// the reverse: 16 registers per thread -> 32 lanes x 16 consecutive columns
__device__ __forceinline__ void tmem_st_x16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- descriptors ------------------------------------------------------------------------
// Shared-memory operand descriptor for a K-major tile stored as rows of 128 bytes (64 fp16)
// with the 128-byte swizzle: 16-byte chunk c of row r sits at r*128 + ((c ^ (r & 7)) << 4),
// 8-row groups 1024 bytes apart, tile base 1024-byte aligned.  Advancing K by 16 elements adds
// 32 bytes to the start address (encoded >> 4, i.e. +2).
__device__ __forceinline__ uint64_t umma_desc_k_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);  // start address, bits [0,14)
    d |= (uint64_t)1 << 16;                         // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;               // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                         // descriptor version (sm_100)
    d |= (uint64_t)2 << 61;                         // layout: SWIZZLE_128B
    return d;
}
// Instruction descriptor, kind::f16: fp16 A and B (both K-major), fp32 D, shape M x N (x16).
__host__ __device__ constexpr uint32_t umma_idesc_f16(uint32_t m, uint32_t n) {
    return (1u << 4)            // D format fp32
           | (0u << 7)          // A fp16
           | (0u << 10)         // B fp16
           | (0u << 15) | (0u << 16)  // A, B K-major
           | ((n >> 3) << 17) | ((m >> 4) << 24);
}

// One lane of a fully converged warp, chosen by the hardware.  Unlike a test of the lane id this tells the
// compiler that exactly one thread runs the guarded code, which lets it keep tcgen05 / TMA operands in uniform
// registers: on B200 an MMA issue loop guarded by elect.sync sustains the tensor pipe's rate through a
// full/empty mbarrier handshake (515 cycles per four 128x256x16 MMAs), the same loop guarded by lane == 0 loses
// about 65 cycles per handshake.
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(pred));
    return pred != 0;
}

// Programmatic dependent launch.  launch_dependents lets the next kernel in the stream (if it was launched with
// the programmatic-serialization attribute) begin its prologue while this grid is still running; grid_dependency_wait
// blocks until the preceding grid has completed and its memory is visible, and is a no-op without such a launch.
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Loads of what a kernel in front may have written.  __ldg and const __restrict__ promise that the data does not change while the kernel is
// there, which began before the one in front had finished: such loads were moved in front of grid_dependency_wait.  These stay behind it, as
// ordinary loads do (the wait is a barrier to them).
__device__ __forceinline__ uint4 ld(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 ld(const uint2* p) {
    uint2 v;
    asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ld(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint16_t ld(const uint16_t* p) {
    uint16_t v;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}

// named barrier among a subset of warps
__device__ __forceinline__ void bar_sync(int id, int nthreads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
// bar_sync that tells every thread whether `pred` holds on all of them
__device__ __forceinline__ bool bar_all(int id, int nthreads, bool pred) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %3, 0;\n\t"
        "bar.red.and.pred q, %1, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r) : "r"(id), "r"(nthreads), "r"((uint32_t)pred) : "memory");
    return r != 0;
}

}  // namespace ptx
