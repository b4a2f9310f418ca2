// sm100.cuh -- thin inline-PTX layer over the Blackwell (sm_100a) primitives the kernels use:
// mbarrier, TMA tiled loads (never with cluster multicast), tcgen05 MMA / commit / TMEM load,
// TMEM allocation, and the shared-memory / instruction descriptors of tcgen05.mma.
//
// Waits on an mbarrier are bounded: one that does not complete within kWaitLimitNs raises a bit in a
// device status word and returns false, so that a logic error shows up as an error code on the
// host instead of a hung GPU.
//
// Three waits of the hardware have no limit and no status bit.  They end because of an order that every kernel keeps:
//   tcgen05.alloc      waits for columns that a CTA of an earlier grid of the stream holds on the SM.  A kernel that takes TMEM lets its successor
//                      start (pdl_release) only behind its own allocation, so a later grid never holds what an earlier one still asks for; and
//                      the earlier grid gives its columns back after bounded waits alone.
//   griddepcontrol.wait  waits for the grid before, which waits for the one before it: back to one that was launched in the ordinary way.
//   barrier.cluster.wait  waits for CTAs that the hardware starts together; each of them arrives on every path, also after an aborted wait.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace spt { namespace sm100 {

constexpr unsigned long long kWaitLimitNs = 2000000000ull;   // 2 s; normal waits are microseconds

// status bits written by kernels (read by sptorch_sync)
constexpr uint32_t kErrProducerWait = 0x1, kErrMmaWait = 0x2, kErrEpilogueWait = 0x4, kErrBadIndex = 0x100;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long globaltimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// CLUSTER: what other CTAs of the cluster sent before the phase completed is visible behind it
template <bool CLUSTER = false>
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    if constexpr (CLUSTER)
        asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t"
            "}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
    else
        asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t"
            "}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
    return ok;
}

// Bounded wait.  `abort_flag` (shared memory) lets one role's failure release the others early.
// The phase is usually complete: that is one test in line.  The spinning lies out of line, because a loop beside the test costs the test its pace: a
// warp that waited, elected and issued four tcgen05.mma of 128 x 16 (64, 128) per turn took 379 (397, 429) cycles a turn with the loop in line,
// 212 (-, 297) with a vote and the loop out of line, and one elected thread that runs the whole loop 171 (-, 261); the four products alone
// take 159 (195, 259).  So producers and MMA issuers are one thread each, and a warp's waits are a vote.
template <bool CLUSTER>
__device__ __forceinline__ bool mbar_spin_here(uint32_t bar, uint32_t parity, volatile int* abort_flag, uint32_t* status, uint32_t code) {
    unsigned long long t0 = globaltimer();
    for (uint32_t spin = 1;; ++spin) {
        if (mbar_try_wait<CLUSTER>(bar, parity)) return true;
        if ((spin & 0xff) == 0) {
            if (*abort_flag) return false;
            if (globaltimer() - t0 > kWaitLimitNs) {
                *abort_flag = 1;
                atomicOr(status, code);
                return false;
            }
        }
    }
}
template <bool CLUSTER>
__device__ __noinline__ bool mbar_spin(uint32_t bar, uint32_t parity, volatile int* abort_flag, uint32_t* status, uint32_t code) {
    return mbar_spin_here<CLUSTER>(bar, parity, abort_flag, status, code);
}
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, uint32_t* status, uint32_t code) {
    return mbar_try_wait<CLUSTER>(bar, parity) || mbar_spin<CLUSTER>(bar, parity, abort_flag, status, code);
}

// for a rare wait with many registers live, which a call would have to save
__device__ __forceinline__ bool mbar_wait_here(uint32_t bar, uint32_t parity, volatile int* abort_flag, uint32_t* status, uint32_t code) {
    return mbar_spin_here<false>(bar, parity, abort_flag, status, code);
}
// a thread that waits by itself, as the issuer of the products does
__device__ __forceinline__ bool wait_alone(uint32_t bar, uint32_t parity, volatile int* abort_flag, uint32_t* status, uint32_t code) { return mbar_wait(bar, parity, abort_flag, status, code); }

// The same for a whole warp: the lanes time themselves, so one may give up while another still sees the phase complete; they go on as one.
template <bool CLUSTER>
__device__ __noinline__ bool mbar_spin_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag, uint32_t* status, uint32_t code) {
    return __all_sync(0xffffffffu, mbar_spin<CLUSTER>(bar, parity, abort_flag, status, code));
}
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag, uint32_t* status, uint32_t code) {
    return __all_sync(0xffffffffu, mbar_try_wait(bar, parity)) || mbar_spin_warp<false>(bar, parity, abort_flag, status, code);
}
// the same with everything in line, for warps with many registers live (a call makes them keep those where a callee must)
__device__ __forceinline__ bool mbar_wait_warp_here(uint32_t bar, uint32_t parity, volatile int* abort_flag, uint32_t* status, uint32_t code) {
    return __all_sync(0xffffffffu, mbar_try_wait(bar, parity) || mbar_spin_here<false>(bar, parity, abort_flag, status, code));
}
// a barrier on which other CTAs of the cluster count what they send: it is visible behind the wait
struct ClusterBar { uint32_t addr; };
__device__ __forceinline__ bool mbar_wait_warp(ClusterBar bar, uint32_t parity, volatile int* abort_flag, uint32_t* status, uint32_t code) {
    return __all_sync(0xffffffffu, mbar_try_wait<true>(bar.addr, parity)) || mbar_spin_warp<true>(bar.addr, parity, abort_flag, status, code);
}

// ---- TMA: tiled load global -> shared, completion on an mbarrier (no multicast, no cache hint) ----
__device__ __forceinline__ void tma_load_4d(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}
// the box's bytes into L2, nothing else
__device__ __forceinline__ void tma_prefetch_l2_4d(const CUtensorMap* map, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global [%0, {%1, %2, %3, %4}];"
                 ::"l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// ---- CTA pairs (cluster of two CTAs sharing one tcgen05.mma, cta_group::2) ----
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// all threads of both CTAs
// The aligned forms want every lane of the warp at the same instruction; a branch before them may have parted the lanes, hence the __syncwarp.
// Two halves: everything before the arrival is visible behind the wait.
__device__ __forceinline__ void cluster_arrive() { __syncwarp(); asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { __syncwarp(); asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() { cluster_arrive(); cluster_wait(); }
// shared::cluster address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa(uint32_t smem_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// the arrival alone, ordering nothing (for a barrier that only keeps CTAs from leaving); lanes may come one by one
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
// 16 bytes into the shared memory of a CTA of the cluster, counted on a barrier of that CTA (both named by shared::cluster addresses)
__device__ __forceinline__ void send16(uint32_t dst, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(dst), "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar) : "memory");
}
__device__ __forceinline__ void send4(uint32_t dst, uint32_t bar, float v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst), "r"(__float_as_uint(v)), "r"(bar) : "memory");
}
// tiled load into this CTA's shared memory whose bytes are counted on an mbarrier that may live in the peer CTA
// (not a multicast: each CTA of the pair loads its own half of the operands)
__device__ __forceinline__ void tma_load_4d_pair(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar_cluster_addr, int c0, int c1, int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}
// TMEM allocation for a pair: the same warp index of BOTH CTAs executes each of these
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_result, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_result), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// ---- TMEM ----
__device__ __forceinline__ void tmem_alloc(uint32_t smem_result, uint32_t ncols) {   // whole warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_result), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {       // whole warp
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// One lane of a converged warp, chosen by the hardware.  Unlike `lane == 0` the result is known to the compiler to hold for exactly
// one thread of a warp-uniform region, so the code under it (descriptor arithmetic, the MMA issue itself) can use the uniform
// datapath instead of moving every operand from a per-thread register first: measured on the attention kernel, whose twelve MMAs
// per key-tile step cost about 100 cycles each to issue under `lane == 0`.
__device__ __forceinline__ bool elect_one_sync() {
    uint32_t pred;
    asm volatile(
        "{\n\t"
        ".reg .pred P1;\n\t"
        "elect.sync _|P1, 0xFFFFFFFF;\n\t"
        "selp.u32 %0, 1, 0, P1;\n\t"
        "}\n"
        : "=r"(pred));
    return pred != 0;
}

// ---- tcgen05.mma, operands in shared memory, accumulator in TMEM ----
// kind::f16 covers f16 and bf16 inputs; kind::tf32 reads f32 containers as tf32.
template <bool TF32>
__device__ __forceinline__ void mma_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    if constexpr (TF32) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n"
            ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
            ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}
// One MMA over the pair: M = 256 (rows 0..127 from this CTA's A tile and TMEM, 128..255 from the peer's), N split the same
// way over the two B tiles; issued by one thread of the even CTA, descriptors are offsets valid in both CTAs.
template <bool TF32>
__device__ __forceinline__ void mma_ss_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    if constexpr (TF32) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n"
            ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
            ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}
// as mma_commit, for pair MMAs; the barrier is named by its shared::cluster address (either CTA of the pair)
__device__ __forceinline__ void mma_commit_pair(uint32_t bar_cluster_addr) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_cluster_addr) : "memory");
}

// arrives (count 1) on the mbarrier once every tcgen05 op issued so far BY THIS THREAD has completed
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp receives lane (base_lane + i)
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
// the same for 8, 16 or 32 columns, by the size of the array
__device__ __forceinline__ void tmem_ld_32xN(uint32_t taddr, uint32_t (&r)[32]) { tmem_ld_32x32(taddr, r); }
__device__ __forceinline__ void tmem_ld_32xN(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_32xN(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// the inverse: thread i of the warp writes 32 consecutive 32-bit columns of lane (base_lane + i)
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
          "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
          "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- descriptors ----
// Shared-memory matrix descriptor for a K-major operand tile stored as rows of exactly 128 bytes with
// the 128-byte swizzle (what a TMA box of {128 B, rows} with SWIZZLE_128B writes).  Fields:
//   [0,14)  start address >> 4          [16,30) leading byte offset >> 4 (unused for swizzled K-major: 1)
//   [32,46) stride byte offset >> 4 = 1024 B between 8-row groups   [46,48) version = 1 on sm_100
//   [61,64) layout type: 2 = SWIZZLE_128B
// Advancing along K inside the 128-byte row by one MMA (32 bytes) adds 2 to the start-address field.
__device__ __forceinline__ uint64_t make_kmajor_sw128_desc(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// Instruction descriptor of tcgen05.mma kind::f16 / kind::tf32, dense, f32 accumulate, both operands K-major:
//   [4,6) D format: 1 = f32    [7,10) A format, [10,13) B format: 1 = bf16, 2 = tf32
//   [15] A major, [16] B major: 0 = K-major    [17,23) N >> 3    [24,29) M >> 4
__host__ __device__ constexpr uint32_t make_idesc(bool tf32, int m, int n) {
    return (1u << 4) | ((tf32 ? 2u : 1u) << 7) | ((tf32 ? 2u : 1u) << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

}}  // namespace spt::sm100
