// PTX wrappers shared by the tensor-core kernels (tcgen05 convolution / matmul and tcgen05 attention): mbarriers
// with bounded waits, TMA tile loads, cluster barriers and distributed shared memory, UMMA descriptors, tcgen05
// issue / commit / load, TMEM release.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace reef {

constexpr int TC_UMMA_M = 128;   // rows of every UMMA tile here = the 128 lanes of tensor memory

// Completion counters: a reduction with release semantics at GPU scope.  Issued by one thread behind a CTA barrier, it
// orders every store of the CTA before the increment and, unlike fence + atomicAdd, waits for no value to come back.
__device__ __forceinline__ void red_release_gpu_add(int* p, int v) {
    asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The completion counter of a best-effort kernel, issued by one thread behind a CTA barrier.  It says that the block ran to its
// end, over whole data if every kernel before it has a full counter too (HybridExecutor::get_be_kernel_offset), and is read behind the kernel's end only (a copy on its stream), which publishes all stores: with release semantics the
// thread waited for the CTA's stores to reach L2 first, in every block between its last store and its exit.
__device__ __forceinline__ void red_relaxed_gpu_add(int* p, int v) {
    asm volatile("red.relaxed.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Every wait is bounded: it gives up after this time (one second; the test of what follows an expired wait takes less).
#ifndef REEF_WAIT_LIMIT_NS
#define REEF_WAIT_LIMIT_NS 1000000000
#endif
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
// The same for data that the other CTAs of the cluster have stored (st_async): acquire at cluster scope.
__device__ __forceinline__ bool mbar_try_cluster(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
// The wait of one thread: false when it gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    unsigned long long t0 = 0;
    for (int i = 0; i < (1 << 26); i++) {
        if (mbar_try(bar, parity)) return true;
        if ((i & 255) == 255) {
            const unsigned long long t = global_ns();
            if (t0 == 0) t0 = t;
            else if (t - t0 > REEF_WAIT_LIMIT_NS) return false;
        }
    }
    return false;
}
// The waits of a whole warp: every lane polls, the warp leaves together (the votes keep its control flow, and with it the
// addresses and descriptors of what it issues next, warp-uniform).
__device__ __forceinline__ bool wait_is_over(uint32_t tries, unsigned long long& t0) {
    const unsigned long long t = global_ns();
    if (t0 == 0) t0 = t;
    return __all_sync(0xffffffffu, t - t0 > REEF_WAIT_LIMIT_NS) || tries >= 1u << 26;
}
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity) {
    unsigned long long t0 = 0;
    for (uint32_t i = 0;; i++) {
        if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
        if ((i & 255) == 255 && wait_is_over(i, t0)) return false;
    }
}
__device__ __forceinline__ bool mbar_wait_cluster_warp(uint32_t bar, uint32_t parity) {
    unsigned long long t0 = 0;
    for (uint32_t i = 0;; i++) {
        if (__all_sync(0xffffffffu, mbar_try_cluster(bar, parity))) return true;
        if ((i & 255) == 255 && wait_is_over(i, t0)) return false;
    }
}
// The wait of the best-effort flavour's MMA warp also ends when `abort_word` (shared memory, written by the TMA producer
// of the same CTA when it saw the preempt flag) becomes non-zero.  0 = phase complete, 1 = gave up, 2 = abort requested.
__device__ __forceinline__ int mbar_wait_abortable_warp(uint32_t bar, uint32_t parity, const volatile uint32_t* abort_word) {
    unsigned long long t0 = 0;
    for (uint32_t i = 0;; i++) {
        if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return 0;
        if (__any_sync(0xffffffffu, *abort_word != 0)) return 2;
        if ((i & 255) == 255 && wait_is_over(i, t0)) return 1;
    }
}
// One look, without the suspension that try_wait may take: for a look ahead at a barrier that may be far from complete.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
// A model constant, requested where this stands: a plain load may be moved down to its first use, behind the waits.
__device__ __forceinline__ float ld_param(const float* p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
// An activation of an earlier kernel, under a per-lane condition: a volatile load stays behind griddepcontrol.wait (__ldg
// promises memory that never changes, and the compiler did move such loads above the wait).  Predicated: as a branch around
// the instruction each of them cost about 30 cycles of a launch's tail.
__device__ __forceinline__ float ld_activation_if(bool c, const float* p) {
    float v;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t@q ld.global.f32 %0, [%1];\n\t}" : "=f"(v) : "l"(p), "r"((int)c));
    return v;
}
// one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* tm, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(tm), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* tm, uint32_t bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(tm), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
// as code of a whole warp, `lead` non-zero in the one lane that issues (see umma_tf32_if)
__device__ __forceinline__ void mbar_expect_tx_if(uint32_t lead, uint32_t bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(bar), "r"(bytes), "r"(lead) : "memory");
}
__device__ __forceinline__ void tma_load_2d_if(uint32_t lead, uint32_t dst, const CUtensorMap* tm, uint32_t bar, int c0, int c1) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
        "@q cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}"
        ::"r"(dst), "l"(tm), "r"(bar), "r"(c0), "r"(c1), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d_if(uint32_t lead, uint32_t dst, const CUtensorMap* tm, uint32_t bar, int c0, int c1, int c2) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %6, 0;\n\t"
        "@q cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n\t}"
        ::"r"(dst), "l"(tm), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void tma_prefetch_3d(const CUtensorMap* tm, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(tm), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// split form: arrive early, wait where the guarantee is needed, so the barrier latency hides behind other work
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
// control-only arrive: what the barrier orders was already observed complete through an mbarrier
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float4 ld_smem_v4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
// Store into the shared memory of a CTA of the cluster, counted in bytes by that CTA's mbarrier.  The source is registers: the
// sender may leave at once, and the receiver is alive until its barrier has seen every byte.
__device__ __forceinline__ void st_async_v4_if(bool c, uint32_t addr, uint32_t bar, const uint32_t* v) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %6, 0;\n\t"
                 "@q st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];\n\t}"
                 ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(bar), "r"((int)c)
                 : "memory");
}
__device__ __forceinline__ void st_smem_v4_if(bool c, uint32_t addr, const uint32_t* v) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t@q st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n\t}"
                 ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"((int)c)
                 : "memory");
}
__device__ __forceinline__ void st_async_u32(uint32_t addr, uint32_t bar, uint32_t v) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(v), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_dsmem_u32(uint32_t addr, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// Shared-memory matrix descriptor, K-major, 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);         // start address >> 4, bits [0,14)
    d |= (uint64_t)1 << 16;                          // leading byte offset (unused with swizzle), bits [16,30)
    d |= (uint64_t)(1024 >> 4) << 32;                // stride byte offset between 8-row groups, bits [32,46)
    d |= (uint64_t)1 << 46;                          // descriptor version for sm_100
    d |= (uint64_t)2 << 61;                          // SWIZZLE_128B
    return d;
}
// Instruction descriptor: D fp32, A/B tf32, both K-major, M=128, N=n.
__device__ __forceinline__ uint32_t umma_idesc_tf32(int n) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TC_UMMA_M >> 4) << 24);
}
__device__ __forceinline__ void umma_tf32(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The same as code of a whole warp: `lead` is non-zero in the one lane that issues.  Predicated, so that the warp's control flow
// stays uniform and the descriptors in uniform registers: the tensor core is then fed at its own rate, measured over resident
// operands as (4096 + 32 N) / 32 cycles per K block of four instructions up to N = 128 (operand reads from shared memory: 160 at
// N = 32, 192 at 64, 256 at 128) and 2 N beyond.  A branch around the instructions, and a look at the barrier between them, cost 307 at
// N = 32 and 332 at 96.
__device__ __forceinline__ void umma_tf32_if(uint32_t lead, uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void umma_commit_if(uint32_t lead, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
        ::"r"(bar), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld4_nowait(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
}
// 32 columns of one TMEM lane per thread; the wait is separate so that several loads can be in flight
__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// by the warp that allocated, after a CTA barrier behind every tcgen05 operation that used the columns
__device__ __forceinline__ void tmem_free(uint32_t tmem, uint32_t cols) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}

}  // namespace reef
