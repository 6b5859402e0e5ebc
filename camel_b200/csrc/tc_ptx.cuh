// Inline-PTX wrappers for the sm_100a features the contraction kernels use: mbarriers with
// BOUNDED waits, TMA tile loads (cp.async.bulk.tensor; every CTA fetches its own tiles), tensor memory (TMEM)
// allocation, tcgen05.mma / commit / ld, and the shared-memory matrix descriptors.
#pragma once

#include <cstdint>

namespace ct {
namespace ptx {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// One lane of a converged warp.  The roles that issue MMAs and copies are entered through this and not through lane == 0: the
// compiler then knows that one thread runs them, and an MMA costs it fewer instructions.  The tensor pipe takes few MMAs ahead,
// so what the issuing thread does between two of them shows: with six 128 x 240 x 16 MMAs (720 clocks), a barrier wait and a
// commit to a stage, another 300 clocks of work are hidden entered so, and none are entered through lane == 0 (1100 clocks a
// stage at 400 of work, 815 so).  256 x 64 x 56 x 56 -> 128, 3 x 3: 504 -> 484 us, 64 x 48 x 57 x 57 -> 96 at stride 2 69.3 -> 65.3,
// 4096 x 784 -> 1024 -> 1024 -> 10 85.8 -> 83.9, bf16 8192^3 1136 -> 1117.
__device__ __forceinline__ bool elect_one() {
    uint32_t pred = 0;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(pred));
    return pred != 0;
}

// ---- mbarrier ---------------------------------------------------------------------------

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// What a wait orders: what this CTA's threads and copies wrote before they arrived; what threads of the whole cluster wrote
// (mbar_arrive_peer_written); or nothing but the execution (mbar_arrive_peer_read: tcgen05.fence does the rest).
enum WaitFor { kCta, kClusterWritten, kClusterRead };
template <WaitFor FOR = kCta>
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
#define CT_TRY_WAIT(SEM)                                                \
    asm volatile(                                                       \
        "{\n\t"                                                         \
        ".reg .pred p;\n\t"                                             \
        "mbarrier.try_wait.parity" SEM ".shared::cta.b64 p, [%1], %2;\n\t" \
        "selp.u32 %0, 1, 0, p;\n\t"                                     \
        "}\n"                                                           \
        : "=r"(ok)                                                      \
        : "r"(bar), "r"(parity)                                         \
        : "memory")
    if (FOR == kClusterWritten)
        CT_TRY_WAIT(".acquire.cluster");
    else if (FOR == kClusterRead)
        CT_TRY_WAIT(".relaxed.cluster");
    else
        CT_TRY_WAIT("");
#undef CT_TRY_WAIT
    return ok != 0;
}

// The same with a time limit for the hardware's own suspension of the thread: a waiting thread
// sleeps until the phase completes (it is woken at once then) or the limit passes, instead of
// coming back after the much shorter system default and polling again.  For roles whose waits are
// long and whose polling would take issue slots from the warps that have work.
__device__ __forceinline__ bool mbar_try_wait_for(uint32_t bar, uint32_t parity, uint32_t limit_ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(limit_ns)
        : "memory");
    return ok != 0;
}

// Wait budget of one barrier wait.  A healthy kernel waits microseconds; the budget only
// exists so that a protocol bug ends as an error status instead of a hung GPU.
constexpr uint64_t kWaitBudgetNs = 1000ull * 1000ull * 1000ull; // 1 s

// Bounded wait.  Returns false when the budget ran out or when another role has already
// given up (*abort_flag != 0); in the first case it raises *abort_flag itself.
template <WaitFor FOR = kCta>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    if (mbar_try_wait<FOR>(bar, parity))
        return true;
    uint64_t t0 = globaltimer_ns();
    for (uint32_t it = 1;; ++it) {
        if (mbar_try_wait<FOR>(bar, parity))
            return true;
        if ((it & 63u) == 0) {
            if (*abort_flag)
                return false;
            if (globaltimer_ns() - t0 > kWaitBudgetNs) {
                *abort_flag = 1;
                return false;
            }
        }
    }
}

// Bounded wait for the patient roles (see mbar_try_wait_for): same contract as mbar_wait.
__device__ __forceinline__ bool mbar_wait_patient(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    if (mbar_try_wait(bar, parity))
        return true;
    uint64_t t0 = globaltimer_ns();
    for (uint32_t it = 1;; ++it) {
        if (mbar_try_wait_for(bar, parity, 20000u))
            return true;
        if (*abort_flag)
            return false;
        if (globaltimer_ns() - t0 > kWaitBudgetNs) {
            *abort_flag = 1;
            return false;
        }
    }
}

// The two for a converged warp: the answer is the same for all lanes, and known to be.
template <WaitFor FOR = kCta>
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    bool got = mbar_try_wait<FOR>(bar, parity);
    if (!__all_sync(0xffffffffu, got))
        got = mbar_wait<FOR>(bar, parity, abort_flag);
    return __all_sync(0xffffffffu, got) != 0;
}
__device__ __forceinline__ bool mbar_wait_patient_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    const bool got = mbar_wait_patient(bar, parity, abort_flag);
    return __all_sync(0xffffffffu, got) != 0;
}

// A wait of several warps: the first of them waits, the others stop at named barrier `id` of `threads` threads, which takes no issue
// slots (an mbarrier wait polls: with eighteen warps of the few-channel convolution waiting by themselves a third of all its
// instructions, 65 of 200 million at 2048 images, were theirs).  All get the same answer, so that all leave when it ran out; `word` holds
// it, two of them in turn.  As bounded as the first warp's wait.
template <typename Wait>
__device__ __forceinline__ bool group_wait(bool waits, Wait wait, volatile int *word, int turn, int id, int threads) {
    if (waits) {
        const bool all = __all_sync(0xffffffffu, wait()) != 0;
        if ((threadIdx.x & 31) == 0)
            word[turn & 1] = all ? 1 : 0;
    }
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
    return __any_sync(0xffffffffu, word[turn & 1]) != 0;
}

// ---- TMA --------------------------------------------------------------------------------

__device__ __forceinline__ void prefetch_tensormap(const void *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// 2-D tile load global -> shared of THIS CTA, completion counted on an mbarrier of this CTA.
// c0 is the innermost (contiguous) coordinate and must make a 16-byte aligned start.
__device__ __forceinline__ void tma_load_2d(
    uint32_t dst_smem, const void *map, uint32_t bar, int32_t c0, int32_t c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];"
        :
        : "r"(dst_smem), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}

__device__ __forceinline__ void tma_load_3d(
    uint32_t dst_smem, const void *map, uint32_t bar, int32_t c0, int32_t c1, int32_t c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5}], [%2];"
        :
        : "r"(dst_smem), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}

// Only c0 carries the 16-byte alignment rule; c1..c3 may be negative or past the end (the
// out-of-range part of the box reads as zero), which is how a convolution's halo is fetched.
__device__ __forceinline__ void tma_load_4d(
    uint32_t dst_smem, const void *map, uint32_t bar, int32_t c0, int32_t c1, int32_t c2, int32_t c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6}], [%2];"
        :
        : "r"(dst_smem), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2),
          "r"(c3)
        : "memory");
}

__device__ __forceinline__ void tma_load_5d(
    uint32_t dst_smem, const void *map, uint32_t bar, int32_t c0, int32_t c1, int32_t c2, int32_t c3, int32_t c4) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
        :
        : "r"(dst_smem), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
        : "memory");
}

// ---- tensor memory ----------------------------------------------------------------------

// Whole-warp instructions (.sync.aligned): call from all 32 lanes of one warp.
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t columns) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem),
                 "r"(columns)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(columns)
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before_sync() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after_sync() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Makes the mbarrier track completion of all MMAs this thread issued so far.
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

// D[tmem] (+)= A[smem] * B[smem]; one thread issues.  accumulate == 0 overwrites D.
__device__ __forceinline__ void mma_tf32(
    uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t"
        "}\n"
        :
        : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_f16(
    uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "}\n"
        :
        : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// ---- CTA pairs (clusters of two CTAs that work on one 256-row tile) ----------------------------
//
// With cta_group::2 one thread of the leader (rank 0) issues MMAs of 256 rows: each CTA of the pair holds
// its 128 rows of A, half of the rows of B and the accumulator of its rows, at the same offsets.

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// cluster_sync in two halves, for threads that need not be converged.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// The address of this CTA's shared-memory location in CTA `rank` of the cluster, and a store of 16 bytes there.
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster_f4(uint32_t cluster_addr, float4 v) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}
// The address of the same shared-memory location in the leader.
__device__ __forceinline__ uint32_t leader_addr(uint32_t addr) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
    return r;
}
// 16 bytes at this CTA's shared-memory offset in CTA `rank` of the cluster.
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr, uint32_t rank) {
    uint32_t r;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(r)
                 : "memory");
    return v;
}
// Arrivals on the leader's barrier.  A warp that has filled its CTA's operands publishes them to the issuer, a thread of the other
// CTA: release at cluster scope, and the issuer waits with kClusterWritten.
__device__ __forceinline__ void mbar_arrive_peer_written(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// A warp that hands back tensor memory publishes nothing: what it has read is in its registers (tcgen05.wait::ld), and tcgen05.fence orders
// that before the arrival; the issuer waits with kClusterRead.  A release would wait until the thread's earlier stores to
// global memory are in L2, 2200 clocks of a tile of the few-channel convolution, whose epilogue stores before it hands back.
__device__ __forceinline__ void mbar_arrive_peer_read(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// Tile load into THIS CTA's shared memory whose bytes are counted on a barrier of this CTA or the leader.
__device__ __forceinline__ void tma_load_2d_pair(
    uint32_t dst_smem, const void *map, uint32_t cluster_bar, int32_t c0, int32_t c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];"
        :
        : "r"(dst_smem), "l"(reinterpret_cast<uint64_t>(map)), "r"(cluster_bar), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void tma_load_5d_pair(
    uint32_t dst_smem, const void *map, uint32_t cluster_bar, int32_t c0, int32_t c1, int32_t c2, int32_t c3, int32_t c4) {
    asm volatile(
        "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
        :
        : "r"(dst_smem), "l"(reinterpret_cast<uint64_t>(map)), "r"(cluster_bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst_smem, uint32_t columns) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(columns)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(columns) : "memory");
}
// Completion of all MMAs of the pair so far, signalled on the barrier at this offset in both CTAs.
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
        "h"((uint16_t)3)
        : "memory");
}
__device__ __forceinline__ void mma_f16_pair(
    uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "}\n"
        :
        : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_tf32_pair(
    uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t"
        "}\n"
        :
        : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// The same for a whole converged warp whose control flow and operands are uniform, of which one lane issues: addresses and
// descriptors then stay in the uniform registers that the instruction reads.  CG: one CTA, or the leader for a pair.
#define CT_MMA_WARP(GROUP, KIND)                                                      \
    asm volatile(                                                                     \
        "{\n\t"                                                                       \
        ".reg .pred p, q;\n\t"                                                        \
        "elect.sync _|q, 0xffffffff;\n\t"                                             \
        "setp.ne.b32 p, %4, 0;\n\t"                                                   \
        "@q tcgen05.mma.cta_group::" GROUP ".kind::" KIND " [%0], %1, %2, %3, p;\n\t" \
        "}\n"                                                                         \
        :                                                                             \
        : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)          \
        : "memory")
template <int CG = 2>
__device__ __forceinline__ void mma_f16_warp(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    if (CG == 2)
        CT_MMA_WARP("2", "f16");
    else
        CT_MMA_WARP("1", "f16");
}
__device__ __forceinline__ void mma_tf32_pair_warp(
    uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    CT_MMA_WARP("2", "tf32");
}
#undef CT_MMA_WARP
// D = A . B + D * 2^-SHIFT (0 .. 15)
template <int SHIFT, int CG>
__device__ __forceinline__ void mma_f16_shifted_warp(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc) {
#define CT_MMA_SHIFTED(GROUP)                                                        \
    asm volatile(                                                                    \
        "{\n\t"                                                                      \
        ".reg .pred p, q;\n\t"                                                       \
        "elect.sync _|q, 0xffffffff;\n\t"                                            \
        "setp.ne.b32 p, 1, 0;\n\t"                                                   \
        "@q tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], %1, %2, %3, p, %4;\n\t" \
        "}\n"                                                                        \
        :                                                                            \
        : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "n"(SHIFT)              \
        : "memory")
    if (CG == 2)
        CT_MMA_SHIFTED("2");
    else
        CT_MMA_SHIFTED("1");
#undef CT_MMA_SHIFTED
}
template <int CG = 2>
__device__ __forceinline__ void tc_commit_warp(uint32_t bar) {
    if (CG == 2)
        asm volatile(
            "{\n\t"
            ".reg .pred q;\n\t"
            "elect.sync _|q, 0xffffffff;\n\t"
            "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t"
            "}\n" ::"r"(bar),
            "h"((uint16_t)3)
            : "memory");
    else
        asm volatile(
            "{\n\t"
            ".reg .pred q;\n\t"
            "elect.sync _|q, 0xffffffff;\n\t"
            "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
            "}\n" ::"r"(bar)
            : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp receives row (lane base + i).
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}

// 32 lanes x 16 columns: for callers that are short of registers.
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void tmem_ld_wait() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---- descriptors ------------------------------------------------------------------------

// Shared-memory matrix descriptor of a K-major operand tile stored as rows of 128 bytes with
// the 128-byte swizzle (what a TMA box of 128-byte rows with SWIZZLE_128B writes): 8-row groups
// 1024 bytes apart.  Fields (bit positions): start address >> 4 [0,14), leading byte offset
// >> 4 [16,30) (unused for swizzled K-major, 1), stride byte offset >> 4 [32,46) = 64,
// descriptor version 1 [46,48), layout type SWIZZLE_128B = 2 [61,64).
__device__ __forceinline__ uint64_t smem_desc_k_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// Same for tiles whose rows are ROW_BYTES = 128 or 64 bytes wide, written by TMA with the
// matching swizzle (SWIZZLE_128B: layout type 2, SWIZZLE_64B: layout type 4); 8-row groups are
// 8 * ROW_BYTES apart.
template <int ROW_BYTES> __device__ __forceinline__ uint64_t smem_desc_k(uint32_t smem_addr) {
    static_assert(ROW_BYTES == 128 || ROW_BYTES == 64, "operand rows are 128 or 64 bytes");
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)((8 * ROW_BYTES) >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)(ROW_BYTES == 128 ? 2 : 4) << 61;
    return d;
}

// Instruction descriptor, dense, float32 accumulator, both operands K-major.
// ab_format: 0 f16, 1 bf16, 2 tf32.  Fields: c format [4,6) = 1 (f32), a format [7,10),
// b format [10,13), n >> 3 [17,23), m >> 4 [24,29).
__host__ __device__ constexpr uint32_t make_idesc(uint32_t ab_format, uint32_t m, uint32_t n) {
    return (1u << 4) | (ab_format << 7) | (ab_format << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

} // namespace ptx
} // namespace ct
