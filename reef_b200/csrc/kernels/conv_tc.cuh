// conv2d / matmul on the 5th-generation tensor cores (tcgen05, TF32 inputs, fp32 accumulate in TMEM).
//
// GEMM view (implicit, no im2col buffer):  D[co][pixel] = sum_k W[co][k] * X[pixel][k]
//   A = weights  OHWI = [Cout][kh*kw*Cin]  : K-major, M = Cout  -> TMEM lanes (128 per tile)
//   B = activations NHWC                    : K-major per filter tap, N = pixels -> TMEM columns
// Both operands are staged by TMA (cp.async.bulk.tensor, 128-byte swizzle) into a shared-memory
// ring; a K block is 32 channels of one filter tap = one 128-byte row per pixel / per output channel.
// Zero padding, ragged tiles and strides are folded into the tensor maps (out-of-bounds boxes read
// zeros; a stride-s conv uses up to s*s maps over the s-strided sub-lattices of the input).
//
// Batch-1 convolutions are tiny GEMMs (N = 49..3136 pixels), far too few tiles for 148 SMs and too
// many weight bytes per tile for one SM's load bandwidth, so K is split across a thread-block
// CLUSTER (1..8 CTAs).  Each CTA accumulates its K range in TMEM and owns a share of the tile's pixels; it
// stores the other ranks' pixels of its partial tile straight from registers into their shared memory
// (st.async, counted by the receiver's mbarrier) and sums its own share over the ranks in rank order 0..S-1 —
// a fixed order, so results are bit-reproducible (no float atomics, no global scratch, no counters to reset when
// a best-effort run is preempted and re-run).
//
// One warp issues TMA, one warp issues tcgen05.mma, all eight warps run the exchange and the epilogue
// (tcgen05.ld -> +residual -> +bias | *gamma+beta -> ReLU -> stores), a thread being one output channel throughout,
// as tensor memory has it.  What bounds it: a launch of a small layer is a chain of latencies (hand-over from the previous grid and
// first K block 1.4 us, the rank's few K blocks, exchange 0.7 us, rows 0.4); a large 3x3 layer is bound by what an SM takes in, 57
// bytes a clock of operands (3x3, 512 channels, 28x28: 646 cycles per K block of 30 KB and two CTAs on an SM, where the
// multiplications need 240) and 16 of partial sums.  Shares stored into the owner replace partials read out of the peers'
// staged tiles between two cluster barriers: 28 pixels over eight ranks 1.65 -> 0.66 us from the accumulator to the last share; with
// multiplications issued at the tensor core's pace, 1x1 1024 -> 256 at 14x14 4.4 -> 3.1 us a launch, 3x3 256 -> 256 5.0 -> 4.0.
// Every mbarrier wait is bounded.  A warp that gave up skips its further waits and sends what it has; the CTA stays until nothing can be
// stored into its shared memory any more (peers' shares, its own loads; bounded again), records the error word, frees its TMEM
// and returns.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "conv_tc_params.h"
#include "tc_common.cuh"

namespace reef {


enum : int { TC_EP_RES = 1, TC_EP_BIAS = 2, TC_EP_GB = 4, TC_EP_RELU = 8, TC_EP_ROUND = 16, TC_EP_GELU = 32 };

// exact-erf GELU (reference: resource/bert/bert.cu:167-173).  Not inlined here on purpose: inlined, the compiler turned
// the uniform `if (gelu)` of the epilogue into straight-line code and every layer paid for erff on each element
// (0.5 us per launch on the row-finishing loop).  Where a whole loop is for GELU layers (tc_finish<.., true>) it is inlined:
// the calls made BERT's 768 -> 3072 matmul at 384 tokens spend 8 us on finishing its rows.
__device__ __forceinline__ float tc_gelu_inline(float v) { return v * (0.5f * erff(v * 0.70710678118654752440f) + 0.5f); }
static __device__ __noinline__ float tc_gelu(float v) { return tc_gelu_inline(v); }

// The tensor core reads only the upper 19 bits of an fp32 operand (truncation, a bias toward zero).  Rounding the stored
// activation to the nearest TF32 value makes the consumer's truncation exact.
__device__ __forceinline__ float4 tc_round4(float4 o) {
    uint32_t u;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(o.x)); o.x = __uint_as_float(u);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(o.y)); o.y = __uint_as_float(u);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(o.z)); o.z = __uint_as_float(u);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(o.w)); o.w = __uint_as_float(u);
    return o;
}

// Branch-free form of (+residual) (+bias | *gamma+beta) (ReLU): r = 0, sc = 1, sh = 0, lo = -inf stand in for
// the absent terms (v + 0 and fma(v, 1, b) are exact, so this equals the conditional form bit for bit).
// The 4 channels of a lane at once: one uniform branch per pixel row instead of one per element.  With GELU: matmul + bias ->
// GELU -> (+residual).
__device__ __forceinline__ float4 tc_epilogue4(float4 v, float4 r, float4 sc, float4 sh, float lo, bool rnd, bool gelu) {
    float4 o;
    if (gelu) {
        o.x = tc_gelu(v.x + sh.x) + r.x; o.y = tc_gelu(v.y + sh.y) + r.y;
        o.z = tc_gelu(v.z + sh.z) + r.z; o.w = tc_gelu(v.w + sh.w) + r.w;
    } else {
        o.x = fmaxf(fmaf(v.x + r.x, sc.x, sh.x), lo); o.y = fmaxf(fmaf(v.y + r.y, sc.y, sh.y), lo);
        o.z = fmaxf(fmaf(v.z + r.z, sc.z, sh.z), lo); o.w = fmaxf(fmaf(v.w + r.w, sc.w, sh.w), lo);
    }
    return rnd ? tc_round4(o) : o;
}

// second output of the dual epilogue: relu(o + b2), rounded like the first when the layer rounds
__device__ __forceinline__ float4 tc_preact(float4 o, float4 b2, bool rnd) {
    float4 r;
    r.x = fmaxf(o.x + b2.x, 0.f); r.y = fmaxf(o.y + b2.y, 0.f); r.z = fmaxf(o.z + b2.z, 0.f); r.w = fmaxf(o.w + b2.w, 0.f);
    return rnd ? tc_round4(r) : r;
}


// Phase trace: compiled in only with -DREEF_DEBUG_AIDS (a development aid; the default build carries no stamps)
#ifdef REEF_DEBUG_AIDS
__device__ __forceinline__ void tc_stamp(const TcParams& P, int slot) {
    if (P.trace != nullptr && blockIdx.x == 0 && blockIdx.y == 0) P.trace[slot] = clock64();
}
// the load of one K block of one rank that is announced and never made: what waits for it gives up
__device__ __forceinline__ bool tc_withheld(const TcParams& P, int i) { return blockIdx.y == 0 && P.withheld_rank == (int)blockIdx.x && P.withheld_load == i; }
// ... and sends its shares this much later
__device__ __forceinline__ void tc_withheld_delay(const TcParams& P) {
    if (P.withheld_delay_ns > 0 && blockIdx.y == 0 && P.withheld_rank == (int)blockIdx.x)
        for (const unsigned long long t = global_ns(); global_ns() - t < (unsigned long long)P.withheld_delay_ns;) __nanosleep(1000);
}
#else
__device__ __forceinline__ void tc_stamp(const TcParams&, int) {}
__device__ __forceinline__ bool tc_withheld(const TcParams&, int) { return false; }
__device__ __forceinline__ void tc_withheld_delay(const TcParams&) {}
#endif

__device__ __forceinline__ float tc_round1(float v) {
    uint32_t u;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(v));
    return __uint_as_float(u);
}

// What a thread finishes pixel groups (of four) with: output channel `co`, every other group of the rank's
// share.  With two warps on a scheduler a hundred instructions of a warp are 0.2 us and more, so what can be worked
// out ahead of the last wait is, and everything per pixel is predicated.
struct TcShare {
    float *out, *out2;         // this channel of the first group's first pixel; eight pixels further per turn.  Pointers: a slice of a
    const float* res;          // wide buffer may lie beyond 2^32 elements
    int count, left;           // groups; pixels from the first group to the end of the share (0: no such channel)
    float sc, sh, b2;          // scale and shift (bias), shift of the second output
    float rpre[2][4];          // residual of the next two groups
};

// Finishes the groups of a share.  The sum of a group over the cluster's ranks 0..S-1 in rank order (a fixed order:
// bit-reproducible) comes from the receive area, `src` being the place of this channel and the first group in the slot of rank 0;
// without a K split it comes from tensor memory, `src` being the first group's column.  Stores and residual loads are 128
// contiguous bytes per warp and pixel.  U groups at a time, so that their loads overlap.
template <int S, int U, bool GELU>
__device__ __forceinline__ void tc_finish(const TcParams& P, TcShare& w, uint32_t src) {
    const uint32_t slot_bytes = (uint32_t)P.gpc * (TC_BM * 16);
    const size_t ocs = (size_t)P.ocs, pcs = (size_t)P.pcs, rcs = (size_t)P.co;
    const bool has_res = P.res != nullptr;
#pragma unroll 1
    for (int k0 = 0; k0 < w.count; k0 += U) {
        float v[U][4], r[U][4];
        uint32_t own[U][4];
        float4 part[U][S];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const bool more = u == 0 || k0 + u < w.count;   // (the share's last turn may be short: a group of it is read again)
            if (S == 1) {
                tmem_ld4_nowait(src + (more ? (uint32_t)u * 8u : 0u), own[u]);
            } else {
#pragma unroll
                for (int q = 0; q < S; q++) part[u][q] = ld_smem_v4(src + (more ? (uint32_t)u * (2 * TC_BM * 16) : 0u) + (uint32_t)q * slot_bytes);
            }
        }
        if (has_res) {   // this turn's was requested two groups ago; the next one's travels beside this turn
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    r[u][i] = w.rpre[u][i];
                    if (U == 1) w.rpre[0][i] = w.rpre[1][i];
                    w.rpre[U == 1 ? 1 : u][i] = ld_activation_if(8 * (u + 2) + i < w.left, w.res + (8 * (u + 2) + i) * rcs);
                }
        }
        if (S == 1) {
            tmem_ld_wait();
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    asm volatile("" : "+r"(own[u][i]));   // (used behind the wait)
                    v[u][i] = __uint_as_float(own[u][i]);
                }
        } else {
#pragma unroll
            for (int u = 0; u < U; u++) {
                v[u][0] = part[u][0].x; v[u][1] = part[u][0].y; v[u][2] = part[u][0].z; v[u][3] = part[u][0].w;
#pragma unroll
                for (int q = 1; q < S; q++) { v[u][0] += part[u][q].x; v[u][1] += part[u][q].y; v[u][2] += part[u][q].z; v[u][3] += part[u][q].w; }
            }
        }
        // (uniform branches around whole turns: an absent term costs nothing)
#define TC_EACH(EXPR)                        \
    do {                                     \
        _Pragma("unroll") for (int u = 0; u < U; u++) _Pragma("unroll") for (int i = 0; i < 4; i++) v[u][i] = (EXPR); \
    } while (0)
        if (GELU) TC_EACH(tc_gelu_inline(v[u][i] + w.sh));
        if (has_res) TC_EACH(v[u][i] + r[u][i]);
        if (!GELU) {
            if (P.ep & TC_EP_GB) TC_EACH(fmaf(v[u][i], w.sc, w.sh));
            else TC_EACH(v[u][i] + w.sh);
        }
        if (P.ep & TC_EP_RELU) TC_EACH(fmaxf(v[u][i], 0.f));
        if (P.ep & TC_EP_ROUND) TC_EACH(tc_round1(v[u][i]));
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (8 * u + i < w.left) w.out[(8 * u + i) * ocs] = v[u][i];
        if (P.out2 != nullptr) {
            TC_EACH(fmaxf(v[u][i] + w.b2, 0.f));
            if (P.ep & TC_EP_ROUND) TC_EACH(tc_round1(v[u][i]));
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (8 * u + i < w.left) w.out2[(8 * u + i) * pcs] = v[u][i];
        }
#undef TC_EACH
        src += S == 1 ? 8u * U : 2u * U * (TC_BM * 16);
        w.left -= 8 * U;
        w.out += 8 * U * ocs;
        w.out2 += 8 * U * pcs;
        w.res += 8 * U * rcs;
    }
}

// Finishes the pixel rows [jb, je) a cluster rank owns after a K split: sums the partials of ranks 0..S-1 in
// rank order (a fixed order: bit-reproducible), applies the epilogue and stores 512-byte rows.  RB rows per warp
// are in flight at a time, RB * SMAX 128-bit loads per lane (16: the kernel is built for two CTAs per SM, so
// a thread has 128 registers).
// The persistent chain kernel's form (partials already in this CTA's shared memory).  The residual was written earlier in
// the SAME launch: it is read at L2 (ld.global.cg), never through the non-coherent path.
template <int RB, int SMAX>
__device__ __forceinline__ void tc_finish_split(const TcParams& P, const float* stage, const float* recv, int S, int split,
                                                int jb, int je, int warp, int cbase, int co, int pix0, float4 sc, float4 sh,
                                                float lo, bool rnd, bool gelu, bool has_res, float4 b2) {
    const float* src[SMAX];
#pragma unroll
    for (int q = 0; q < SMAX; q++)
        src[q] = (q == split) ? stage + (size_t)jb * TC_BM + cbase
                              : recv + (size_t)(q < S ? (q < split ? q : q - 1) : 0) * P.cpc_max * TC_BM + cbase;
    for (int jbase = warp; jbase < je - jb; jbase += 8 * RB) {
        float4 part[RB][SMAX], rv[RB];
#pragma unroll
        for (int u = 0; u < RB; u++) {
            const int jr = jbase + 8 * u;   // row within this rank's slice
            rv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (jr < je - jb) {
#pragma unroll
                for (int q = 0; q < SMAX; q++)
                    if (q < S) part[u][q] = *reinterpret_cast<const float4*>(src[q] + (size_t)jr * TC_BM);
                if (has_res) rv[u] = __ldcg(reinterpret_cast<const float4*>(P.res + (size_t)(pix0 + jb + jr) * P.co + co));
            }
        }
#pragma unroll
        for (int u = 0; u < RB; u++) {
            const int jr = jbase + 8 * u;
            if (jr < je - jb) {
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int q = 0; q < SMAX; q++)   // fixed rank order: deterministic sum
                    if (q < S) { v.x += part[u][q].x; v.y += part[u][q].y; v.z += part[u][q].z; v.w += part[u][q].w; }
                const float4 o = tc_epilogue4(v, rv[u], sc, sh, lo, rnd, gelu);
                *reinterpret_cast<float4*>(P.out + (size_t)(pix0 + jb + jr) * P.ocs + P.ooff + co) = o;
                if (P.out2 != nullptr) *reinterpret_cast<float4*>(P.out2 + (size_t)(pix0 + jb + jr) * P.pcs + P.poff + co) = tc_preact(o, b2, rnd);
            }
        }
    }
}

// BE = best-effort flavour (reference wrapper contract: script/best_effort_kernel.py:22-33, with the polls the
// reference gets for free from killing wavefronts): the preempt flag is read at block entry and, by the TMA producer,
// at the head of its refill loop (every 4th K block).  A CTA that saw the flag stops loading and lets the tensor core
// finish what has landed; it takes part in the exchange all the same, each rank sending along what it saw, and if any
// rank stopped, ALL ranks skip the stores and the completion counter — the kernel is idempotent, so it is simply
// launched again later.  The real-time flavour carries none of this.
template <bool BE, int S>
__global__ void __launch_bounds__(TC_THREADS, 2) reef_conv_tc_kernel(const __grid_constant__ TcParams P) {
    extern __shared__ __align__(16) unsigned char tc_smem_raw[];
    // stage buffers need 1024-byte alignment (swizzle atom); carve barriers behind them
    const uint32_t raw = smem_u32(tc_smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* smem = tc_smem_raw + (base - raw);
    const uint32_t stage_bytes = TC_A_BYTES + (uint32_t)P.n_mma * 128u;
    // the control words sit behind the data region (stage ring, reused by the epilogue's staging + exchange area)
    const uint32_t ctrl = base + (uint32_t)P.region_bytes;
    const int NS = P.stages;   // ring depth of this launch (<= TC_MAX_STAGES)
    const uint32_t bar_full = ctrl, bar_empty = ctrl + 8 * TC_MAX_STAGES, bar_acc = ctrl + 16 * TC_MAX_STAGES, bar_recv = bar_acc + 8;
    volatile uint32_t* s_tmem = reinterpret_cast<volatile uint32_t*>(smem + P.region_bytes + 16 * TC_MAX_STAGES + 16);
    volatile uint32_t* s_flags = s_tmem + 1;    // [0] abort (preempt flag seen by this CTA), [1] K blocks whose loads were issued when
                                                //  the producer stopped, [2..9] what the ranks of the cluster saw (best-effort flavour)

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // (known to be warp-uniform)
    // best-effort flavour: the poll at block entry is issued first, so that its latency hides behind the set-up
    int flag0 = 0;
    if (BE && tid == 0) flag0 = *reinterpret_cast<const volatile int*>(P.preempt_flag);
    if (tid == 0) tc_stamp(P, 0);
    // grid = (K splits = cluster, tiles of this launch); a launch may cover a sub-range of the tiles
    const int split = blockIdx.x;
    const int tile = P.tile_begin + (int)blockIdx.y;
    const int tile_n = tile % P.n_tiles, tile_m = tile / P.n_tiles;
    const int kb_begin = split * P.kb_per_split;
    const int kb_end = min(kb_begin + P.kb_per_split, P.kb_total);
    const int nkb = kb_end - kb_begin;

    // spatial tiles: tile_n -> (row group ty, row piece tx); tx > 0 only where a row is wider than a tile
    const int tile_y = P.xsplit > 1 ? tile_n / P.xsplit : tile_n, tile_x = P.xsplit > 1 ? tile_n - tile_y * P.xsplit : 0;
    const int pix0 = P.spatial ? tile_y * P.rows * P.wo + tile_x * P.xw : tile_n * P.n_valid;
    const int m0 = tile_m * TC_BM;
    // columns of this tile that are real pixels, and its real output channels
    const int n_lim = P.xsplit > 1 ? min(P.xw, P.wo - tile_x * P.xw) : min(P.n_valid, P.ptot - pix0);
    const int co_lim = min(TC_BM, P.co - m0);
    // the share of this rank: pixel groups (of four) [grp0, grp0 + mg)
    const int groups = (n_lim + 3) >> 2, gpc = P.gpc;
    const int grp0 = split * gpc, mg = max(0, min(gpc, groups - grp0));
    const uint32_t recv_bytes = (uint32_t)((S - 1) * (mg * co_lim * 16 + (BE ? 4 : 0)));   // from the other ranks

    if (tid == 0) {
        for (int s = 0; s < NS; s++) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_acc, 1);
        mbar_init(bar_recv, 1);
        s_flags[0] = (uint32_t)(flag0 != 0);
        s_flags[1] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (recv_bytes != 0) mbar_expect_tx(bar_recv, recv_bytes);
        asm volatile("prefetch.tensormap [%0];" ::"l"(&P.tm_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&P.tm_x[0]) : "memory");
    }
    // The warp that allocates tensor memory frees it: one of the half that has fewer groups to finish (none, often)
    const int awarp = S > 1 && (grp0 & 1) == 0 ? 5 : 1;
    if (warp == awarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)s_tmem)),
                     "r"((uint32_t)P.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *s_tmem;
    if (tid == 0) tc_stamp(P, 1);   // set-up done (barriers, TMEM)
    // "my receive area may be written": where it is apart from the stage ring, from here on (the barrier's latency then hides
    // behind the main loop); where it lies over the ring, behind the accumulator
    if (S > 1 && !P.recv_late) cluster_arrive();

    bool ok = true;                             // no wait of this warp has expired; one that has ends the others

    // best-effort flavour: what this CTA saw at entry.  Nothing is loaded then; the cluster agrees at its first barrier.
    const bool abort0 = BE && s_flags[0] != 0;

    {
        // ---------------- TMA producer, part 1: fill the ring (no waits) ----------------
        // Warp 0 refills the ring and warp 1 issues the multiplications as whole warps: control flow, addresses and
        // descriptors are warp-uniform (uniform registers), one elected lane executes each instruction.  As code of a
        // single thread every instruction had its operands moved into uniform registers first: 540 cycles per K block in
        // the multiplication loop, whatever the tile's width.
        const uint32_t tx = (uint32_t)P.load_bytes;
        const int first = nkb < NS ? nkb : NS;
        if (warp == 0) {
            // The first loads: one lane per stage.  Weights do not depend on the previous kernel and are requested before
            // the dependency wait, activations after it, their coordinates worked out before it, so that only the copy
            // instruction itself is left on the critical path (30 cycles a lane; 90 with the coordinates in line).
            const CUtensorMap* bmap = &P.tm_x[0];
            int bc0 = 0, bc1 = tile_n * P.n_valid, bc2 = 0;
            if (lane < first && !abort0) {
                const int kb = kb_begin + lane, t = P.cblocks == 1 ? kb : (int)__umulhi((unsigned)kb, P.cb_magic);
                bc0 = (kb - t * P.cblocks) * TC_BK;
                mbar_expect_tx(bar_full + 8 * lane, tx);
                if (!tc_withheld(P, lane)) tma_load_3d(base + lane * stage_bytes, &P.tm_w, bar_full + 8 * lane, bc0, t, m0);
                if (P.spatial) {
                    bmap = &P.tm_x[P.tap_map[t]];
                    bc1 = tile_x * P.xw + P.tap_qx[t];
                    bc2 = tile_y * P.rows + P.tap_qy[t];
                }
            }
            // Weights of the K blocks beyond the ring: into L2, each once among the tiles that share them.  A stage freed by the
            // multiplications is refilled from there in half the time that it takes from HBM (2 to 3 % of a replay of ResNet-152,
            // BERT-base, VGG-16 or DenseNet-201).
            if (!abort0)
                for (int i = first + lane; i < nkb; i += 32) {
                    const int kb = kb_begin + i, t = P.cblocks == 1 ? kb : (int)__umulhi((unsigned)kb, P.cb_magic);
                    if (P.n_tiles == 1 || i % P.n_tiles == tile_n) tma_prefetch_3d(&P.tm_w, (kb - t * P.cblocks) * TC_BK, t, m0);
                }
            asm volatile("griddepcontrol.wait;" ::: "memory");
            // Only now may the next kernel of the stream begin its prologue (set-up, weight loads).  Released
            // any earlier, a chain of these kernels runs ahead without bound and parks its blocks on every SM;
            // in this order at most two grids of a chain are resident and the other SM slots stay free for
            // best-effort kernels.  One thread per CTA executing the instruction counts for the CTA.
            asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            if (lane < first && !abort0 && !tc_withheld(P, lane)) {
                const uint32_t bdst = base + lane * stage_bytes + TC_A_BYTES;
                if (P.spatial) tma_load_3d(bdst, bmap, bar_full + 8 * lane, bc0, bc1, bc2);
                else tma_load_2d(bdst, bmap, bar_full + 8 * lane, bc0, bc1);
            }
            __syncwarp();
            if (lane == 0) tc_stamp(P, 2);   // ring filled (loads issued)
        }
        __syncwarp();

        // warp w reads TMEM lanes 32*(w%4).., its hardware quadrant: a thread is output channel `row` of the tile.  Its epilogue
        // parameters are model constants, requested right after the first loads, so that their latency is long gone when the
        // accumulator is ready.
        const int quad = warp & 3, half = warp >> 2;
        const int row = quad * 32 + lane;
        const int co = m0 + row;
        const bool cvalid = row < co_lim;
        TcShare w;
        w.sc = 1.f; w.sh = 0.f; w.b2 = 0.f;
        if (cvalid) {
            if (P.ep & TC_EP_GB) {
                w.sc = ld_param(P.gamma + co);
                w.sh = ld_param(P.beta + co);
            } else if (P.ep & TC_EP_BIAS) {
                w.sh = ld_param(P.bias + co);
            }
            if (P.bias2 != nullptr) w.b2 = ld_param(P.bias2 + co);
        }
        const bool gelu = (P.ep & TC_EP_GELU) != 0;

        if (warp == 0) {
            // ---------------- TMA producer, part 2: refill stages as the MMAs release them ----------------
            // (stage index and phase parity are carried along: a division by the runtime ring depth per K block
            // is dozens of cycles on this critical path)
            int s = first == NS ? 0 : first;      // first < NS only when nkb < NS, and then this loop does not run
            uint32_t par = 0;                      // parity of the "empty" phase awaited: ((i / NS) - 1) & 1
            int issued = abort0 ? 0 : first;       // K blocks whose loads are out
            bool stop = abort0;
            // filter tap and channel block of the next K block (2^32 / 1 does not fit the magic: one channel block per tap is a copy)
            int tap = P.cblocks == 1 ? kb_begin + first : (int)__umulhi((unsigned)(kb_begin + first), P.cb_magic);
            int cb = kb_begin + first - tap * P.cblocks;
            const uint32_t lead = elect_one() ? 1u : 0u;
            // A second look at the preempt flag, behind the dependency wait: a best-effort kernel queued behind a
            // running one is resident early (programmatic dependent launch) and made its entry poll long before its
            // predecessor finished, possibly before the flag went up.  Its first loads are out (their barriers were
            // armed for both operands, so the activation loads had to follow the weight loads); it issues no more, and
            // the MMA warp only waits for those to land.  Every look is taken four K blocks after its load was issued: waited
            // for in place, the trip to L2 stood between the multiplications (0.6 us a launch, 1.6 in BERT's matmuls).
            int f = 0;
            if (BE) f = *reinterpret_cast<const volatile int*>(P.preempt_flag);
            for (int i = first; i < nkb && ok && !stop; i++) {
                // coordinates are worked out ahead of the wait for a free stage: the per-tap sub-lattice and offsets come from a
                // host table
                const int c0 = cb * TC_BK, t = tap;
                int c1 = tile_n * P.n_valid, c2 = 0, map = 0;
                if (P.spatial) {
                    map = P.tap_map[t];
                    c1 = tile_x * P.xw + P.tap_qx[t];
                    c2 = tile_y * P.rows + P.tap_qy[t];
                }
                if (++cb == P.cblocks) { cb = 0; tap++; }
                ok = mbar_wait_warp(bar_empty + 8 * s, par);
                if (!ok) break;
                if (BE && ((i - first) & 3) == 3) {   // loop-head poll of the preempt flag
                    if (__any_sync(0xffffffffu, f != 0)) { stop = true; break; }
                    f = *reinterpret_cast<const volatile int*>(P.preempt_flag);
                }
                const uint32_t dst = base + s * stage_bytes, bar = bar_full + 8 * s;
                mbar_expect_tx_if(lead, bar, tx);
                if (!tc_withheld(P, i)) {
                    tma_load_3d_if(lead, dst, &P.tm_w, bar, c0, t, m0);
                    if (P.spatial) tma_load_3d_if(lead, dst + TC_A_BYTES, &P.tm_x[map], bar, c0, c1, c2);
                    else tma_load_2d_if(lead, dst + TC_A_BYTES, &P.tm_x[0], bar, c0, c1);
                }
                issued++;
                if (++s == NS) { s = 0; par ^= 1u; }
            }
            if (BE && !stop) stop = __any_sync(0xffffffffu, f != 0);
            if (lane == 0) s_flags[1] = (uint32_t)issued;     // first how far the loads got, then the request to stop
            if (BE && stop && lane == 0) {
                __threadfence_block();
                s_flags[0] = 1;
            }
            __syncwarp();
            // (a wait that expired here leaves the multiplications, and with them the accumulator's barrier, incomplete)
        } else if (warp == 1) {
            // ---------------- MMA issuer ----------------
            // The next stage's barrier is looked at before this stage's multiplications are issued, and those are predicated
            // on the issuing lane instead of branched around: the loop then runs at the tensor core's pace (umma_tf32_if).
            bool halted = false;
            const uint32_t idesc = umma_idesc_tf32(P.n_mma), lead = elect_one() ? 1u : 0u;
#ifdef REEF_DEBUG_AIDS
            const bool tr = lane == 0 && P.trace != nullptr && blockIdx.x == 0 && blockIdx.y == 0;
#endif
            int s = 0;
            uint32_t par = 0;
            uint64_t da = umma_desc_sw128(base);
            bool ready = false;
            for (int i = 0; i < nkb; i++) {
                if (!ready) {
                    if (BE) {
                        const int w = mbar_wait_abortable_warp(bar_full + 8 * s, par, &s_flags[0]);
                        if (w == 2) {
                            // The producer stopped.  Loads it had issued may still be in flight: they must have landed
                            // before this CTA leaves or reuses its shared memory, so their barriers are awaited (bounded)
                            // without multiplying.
                            __threadfence_block();
                            const int issued = __shfl_sync(0xffffffffu, (int)s_flags[1], 0);
                            for (; i < issued && ok; i++) {
                                ok = mbar_wait_warp(bar_full + 8 * s, par);
                                if (++s == NS) { s = 0; par ^= 1u; }
                            }
                            halted = true;
                            break;
                        }
                        ok = w == 0;
                    } else {
                        ok = mbar_wait_warp(bar_full + 8 * s, par);
                    }
                    if (!ok) break;
                }
#ifdef REEF_DEBUG_AIDS
                if (tr && i == 0) P.trace[4] = clock64();          // first K block landed
                if (tr && i == nkb - 1) P.trace[5] = clock64();    // last K block landed
#endif
                const int s2 = s + 1 == NS ? 0 : s + 1;
                const uint32_t par2 = s2 == 0 ? par ^ 1u : par;
                const bool next = mbar_test(bar_full + 8 * s2, par2);
                const uint64_t db = da + (uint64_t)(TC_A_BYTES >> 4);
                // one tcgen05.mma covers K = 8 tf32 = 32 bytes
#pragma unroll
                for (int k = 0; k < TC_BK / 8; k++)
                    umma_tf32_if(lead, tmem, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (i > 0 || k > 0) ? 1u : 0u);
                if (i + NS < nkb) umma_commit_if(lead, bar_empty + 8 * s);   // frees the stage, where it is refilled, once these MMAs have read it
                ready = __all_sync(0xffffffffu, next);
                da = s2 == 0 ? umma_desc_sw128(base) : da + (uint64_t)(stage_bytes >> 4);
                s = s2;
                par = par2;
            }
            // complete, or stopped early: the accumulator's barrier completes when the multiplications issued so far have
            if (ok) umma_commit_if(lead, bar_acc);
        }
        __syncwarp();
        if (warp != 0) asm volatile("griddepcontrol.wait;" ::: "memory");
        // this half's groups of the share: every other one
        const int gfirst = grp0 + ((grp0 ^ half) & 1);
        w.count = max(0, (grp0 + mg - gfirst + 1) >> 1);
        w.left = cvalid && w.count > 0 ? min(n_lim, (grp0 + mg) * 4) - gfirst * 4 : 0;
        w.out = P.out + ((size_t)(pix0 + gfirst * 4) * P.ocs + P.ooff + co);
        w.out2 = P.out2 + ((size_t)(pix0 + gfirst * 4) * P.pcs + P.poff + co);
        w.res = P.res + ((size_t)(pix0 + gfirst * 4) * P.co + co);
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int i = 0; i < 4; i++) w.rpre[u][i] = ld_activation_if(P.res != nullptr && 8 * u + i < w.left, w.res + (size_t)(8 * u + i) * P.co);

        // The exchange: this half's groups of the tile leave tensor memory four at a time for the owner's shared memory, slot `split`
        // there; an own group goes into the own slot (the thread that finishes a group is the one that put it there).  The next
        // rank's leave first, so that the ranks do not all store to the same one.  Where a turn's groups go is worked out ahead of
        // it, for the first turn ahead of the accumulator.
        const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16), recv = base + (uint32_t)P.recv_offset;
        const int turns = (groups - half + 1) >> 1;
        int rot = (grp0 + mg - half + 1) >> 1;
        if (rot >= turns) rot = 0;
        uint32_t col[4], dst[4], bar[4];   // bar = 0: an own group; dst = 0: none
        auto route = [&](int t0) {
            const uint32_t place = (uint32_t)P.recv_offset + (uint32_t)(split * gpc * TC_BM + row) * 16u;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int t = t0 + u, g = half + 2 * (t >= turns ? 0 : t + rot < turns ? t + rot : t + rot - turns);
                const int owner = (int)(((uint32_t)g * P.gpc_magic) >> 16);
                const uint32_t off = place + (uint32_t)(g - owner * gpc) * (TC_BM * 16), peer = owner == split ? base : mapa_shared(base, (uint32_t)owner);
                col[u] = taddr + (uint32_t)g * 4u;
                dst[u] = cvalid && t < turns ? peer + off : 0u;
                bar[u] = owner != split && dst[u] != 0 ? peer + (bar_recv - base) : 0u;
            }
        };
        if (S > 1) {
            route(0);
            if (!P.recv_late) cluster_wait();           // every rank's receive area may be written
        }

        // ---------------- exchange and epilogue: all eight warps ----------------
        ok = ok && mbar_wait_warp(bar_acc, 0);
        tc_withheld_delay(P);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // best-effort flavour: behind this barrier the producer and the MMA warp are past their loops, the flag word is final
        if (BE) __syncthreads();
        bool abort_all = BE && s_flags[0] != 0;
        if (tid == 0) tc_stamp(P, 6);   // accumulator complete
        if (S > 1) {
            if (P.recv_late) {
                cluster_arrive_relaxed();   // (what it orders, the reads of the ring, was seen complete through the accumulator's barrier)
                cluster_wait();
            }
            if (tid == 0) tc_stamp(P, 3);
            // what this rank saw, to every other rank (ahead of the shares: the slowest store is the last)
            if (BE && warp == 7 && lane < S && lane != split) {
                const uint32_t peer = mapa_shared(base, (uint32_t)lane);
                st_async_u32(peer + (smem_u32((const void*)&s_flags[2]) - base) + (uint32_t)split * 4u, peer + (bar_recv - base), abort_all || !ok ? 1u : 0u);
            }
            __syncwarp();
            // (A rank that gave up sends what it has: the receivers count bytes.  The result of a preempted launch is stored by
            // none of them, that of a failed one means nothing: the error word says so.)
            if (quad * 32 < co_lim) {
#pragma unroll 1
                for (int t0 = 0; t0 < turns;) {
                    uint32_t v[4][4];
#pragma unroll
                    for (int u = 0; u < 4; u++) tmem_ld4_nowait(col[u], v[u]);
                    tmem_ld_wait();
#pragma unroll
                    for (int u = 0; u < 4; u++) {
#pragma unroll
                        for (int i = 0; i < 4; i++) asm volatile("" : "+r"(v[u][i]));   // (used behind the wait)
                        st_async_v4_if(bar[u] != 0, dst[u], bar[u], v[u]);
                        st_smem_v4_if(bar[u] == 0 && dst[u] != 0, dst[u], v[u]);
                    }
                    t0 += 4;
                    if (t0 < turns) route(t0);
                }
            }
            // the accumulator is out of tensor memory
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if (warp != awarp) {
                asm volatile("bar.arrive 1, 256;" ::: "memory");
            } else if (w.count == 0) {
                asm volatile("bar.sync 1, 256;" ::: "memory");
                tmem_free(tmem, (uint32_t)P.tmem_cols);
            }
            if (tid == 0) tc_stamp(P, 7);   // shares sent
            // A rank whose shares are there leaves by itself: nothing more will be stored into its shared memory.  One that gave
            // up stays until every warp of the cluster is past its stores, each of them after bounded waits, and these
            // have landed.  (Only then does anybody wait for this barrier; to arrive costs nothing that could be measured.)
            cluster_arrive_relaxed();
            if (recv_bytes != 0) {
                ok = ok && mbar_wait_cluster_warp(bar_recv, 0);
                if (!ok) {
                    cluster_wait();
                    mbar_wait_cluster_warp(bar_recv, 0);
                }
            }
            if (BE) {
                // every rank has the words of all the others: all take the same exit
                if (__any_sync(0xffffffffu, lane < S && lane != split && s_flags[2 + lane] != 0)) abort_all = true;
            }
        }
        if (!ok && P.error_word) *reinterpret_cast<volatile int*>(P.error_word) = 1;
        if (tid == 0) tc_stamp(P, 8);       // shares received
        if (ok && !abort_all && quad * 32 < co_lim) {
            const uint32_t src = S == 1 ? taddr + (uint32_t)gfirst * 4u : recv + (uint32_t)((gfirst - grp0) * TC_BM + row) * 16u;
            constexpr int U = S <= 2 ? 2 : 1;
            if (gelu) tc_finish<S, U, true>(P, w, src);
            else tc_finish<S, U, false>(P, w, src);
        }
        if (tid == 0) tc_stamp(P, 9);   // rows finished
        if (BE && abort_all && tid == 0 && P.stamps != nullptr) {
            // measurement only: when this block saw the preempt flag and left (device clock)
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            atomicMin(&P.stamps[0], t);
            atomicMax(&P.stamps[1], t);
        }
        if (P.task_slot != nullptr && __syncthreads_and(ok && !abort_all) && tid == 0) red_relaxed_gpu_add(P.task_slot, 1);
        // (A rank leaves without waiting for its peers: what it sent them is on its way, and nobody reads its shared memory.)
        if (S == 1) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if (warp != awarp) asm volatile("bar.arrive 1, 256;" ::: "memory");
        }
        if (warp == awarp && !(S > 1 && w.count == 0)) {
            asm volatile("bar.sync 1, 256;" ::: "memory");
            tmem_free(tmem, (uint32_t)P.tmem_cols);
        }
        // a CTA that gave up leaves no load behind that could still write into its shared memory (one limit for all of them)
        if (!ok && warp == 0) {
            const int issued = (int)s_flags[1];
            bool landed = true;
            for (int i = max(0, issued - NS); i < issued && landed; i++) landed = mbar_wait_warp(bar_full + 8 * (i % NS), (uint32_t)(i / NS) & 1u);
        }
    }

    if (tid == 32) tc_stamp(P, 10);   // leaving
}

}  // namespace reef
