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
// CLUSTER (1..8 CTAs).  Each CTA accumulates its K range in TMEM, parks the partial tile in its own
// shared memory, and after a cluster barrier every CTA sums a slice of the tile over all ranks through
// distributed shared memory in rank order 0..S-1 — a fixed order, so results are bit-reproducible (no
// float atomics, no global scratch, no counters to reset when a best-effort run is preempted and re-run).
//
// One warp issues TMA, one warp issues tcgen05.mma, all eight warps run the epilogue
// (tcgen05.ld -> +residual -> +bias | *gamma+beta -> ReLU -> coalesced 512-byte rows, four output
// channels per lane).  What bounds it: a launch of a few microseconds is a chain of latencies (hand-over from
// the previous grid 1.7 us, first K block 0.3 us, cluster barrier 0.6 us, rows 1 us) around a main loop that
// takes about 57 bytes a clock into an SM.  Issue by whole warps and the remote-load epilogue took the replay
// of ResNet-152 from 827 to 760 us, Inception-v3's from 377 to 338 us, BERT's (128 tokens) from 593 to 560 us.
// Every mbarrier wait is bounded: on expiry the kernel records an error word,
// skips further waits, still joins every cluster barrier, frees its TMEM and returns.
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
// (0.5 us per launch on the row-finishing loop).  Where a whole loop is for GELU layers (tc_finish_rows) it is inlined:
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
#else
__device__ __forceinline__ void tc_stamp(const TcParams&, int) {}
#endif

// Finishes the pixel rows [jb, je) this CTA owns: row jb + i of the accumulator is summed over the staged tiles of the
// cluster's ranks 0..S-1 in rank order (a fixed order: bit-reproducible), read from distributed shared memory; then the
// epilogue, and a 512-byte row is stored.  A warp takes every 8th row and RB of them at a time, RB * SMAX 128-bit loads per
// lane in flight (16: the kernel is built for two CTAs per SM, so a thread has 128 registers).
template <int RB, int SMAX, bool GELU>
__device__ __forceinline__ void tc_finish_rows(const TcParams& P, uint32_t stage, int S, int jb, int je, int warp, int cbase, int co, int pix0,
                                               float4 sc, float4 sh, float lo, bool rnd, bool has_res, float4 b2, const float4* rpre) {
    uint32_t src[SMAX];
#pragma unroll
    for (int q = 0; q < SMAX; q++) {
        const uint32_t own = stage + (uint32_t)(jb * TC_BM + cbase) * 4u;
        src[q] = SMAX == 1 ? own : mapa_shared(own, (uint32_t)(q < S ? q : 0));
    }
    for (int jbase = warp; jbase < je - jb; jbase += 8 * RB) {
        float4 part[RB][SMAX], rv[RB];
#pragma unroll
        for (int u = 0; u < RB; u++) {
            const int jr = jbase + 8 * u;   // row within this CTA's share
            rv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (jr < je - jb) {
#pragma unroll
                for (int q = 0; q < SMAX; q++)
                    if (q < S) part[u][q] = SMAX == 1 ? ld_smem_v4(src[q] + (uint32_t)jr * TC_BM * 4u) : ld_dsmem_v4(src[q] + (uint32_t)jr * TC_BM * 4u);
                if (has_res) rv[u] = (u < 2 && jbase == warp) ? rpre[u & 1] : ld_activation(P.res + (size_t)(pix0 + jb + jr) * P.co + co);
            }
        }
#pragma unroll
        for (int u = 0; u < RB; u++) {
            const int jr = jbase + 8 * u;
            if (jr < je - jb) {
                float4 v = part[u][0];
#pragma unroll
                for (int q = 1; q < SMAX; q++)   // fixed rank order: deterministic sum
                    if (q < S) { v.x += part[u][q].x; v.y += part[u][q].y; v.z += part[u][q].z; v.w += part[u][q].w; }
                float4 o;
                if (GELU) {
                    o.x = tc_gelu_inline(v.x + sh.x) + rv[u].x; o.y = tc_gelu_inline(v.y + sh.y) + rv[u].y;
                    o.z = tc_gelu_inline(v.z + sh.z) + rv[u].z; o.w = tc_gelu_inline(v.w + sh.w) + rv[u].w;
                    if (rnd) o = tc_round4(o);
                } else {
                    o = tc_epilogue4(v, rv[u], sc, sh, lo, rnd, false);
                }
                *reinterpret_cast<float4*>(P.out + (size_t)(pix0 + jb + jr) * P.ocs + P.ooff + co) = o;
                if (P.out2 != nullptr) *reinterpret_cast<float4*>(P.out2 + (size_t)(pix0 + jb + jr) * P.pcs + P.poff + co) = tc_preact(o, b2, rnd);
            }
        }
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
// at the head of its refill loop (every 4th K block).  A CTA that saw the flag stops loading, lets the tensor core
// finish what has landed, and takes part in every cluster barrier; at the first barrier the ranks of a cluster
// exchange what they saw, and if any rank stopped, ALL ranks skip the exchange, the stores and the completion counter —
// the kernel is idempotent, so it is simply launched again later.  The real-time flavour carries none of this.
template <bool BE>
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
    const uint32_t bar_full = ctrl, bar_empty = ctrl + 8 * TC_MAX_STAGES, bar_acc = ctrl + 16 * TC_MAX_STAGES;
    volatile uint32_t* s_tmem = reinterpret_cast<volatile uint32_t*>(smem + P.region_bytes + 16 * TC_MAX_STAGES + 16);
    volatile uint32_t* s_flags = s_tmem + 1;    // [0] abort (preempt flag seen by this CTA), [1] wait expired,
                                                //  [2] K blocks whose loads were issued when the producer stopped

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
    const int S = P.splits;
    const int kb_begin = split * P.kb_per_split;
    const int kb_end = min(kb_begin + P.kb_per_split, P.kb_total);
    const int nkb = kb_end - kb_begin;

    if (tid == 0) {
        for (int s = 0; s < NS; s++) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_acc, 1);
        s_flags[0] = (uint32_t)(flag0 != 0);
        s_flags[1] = 0;
        s_flags[2] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&P.tm_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&P.tm_x[0]) : "memory");
    }
    if (warp == 1) {
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

    // spatial tiles: tile_n -> (row group ty, row piece tx); tx > 0 only where a row is wider than a tile
    const int tile_y = P.xsplit > 1 ? tile_n / P.xsplit : tile_n, tile_x = P.xsplit > 1 ? tile_n - tile_y * P.xsplit : 0;
    const int pix0 = P.spatial ? tile_y * P.rows * P.wo + tile_x * P.xw : tile_n * P.n_valid;
    // columns of this tile that are real pixels
    const int n_lim = P.xsplit > 1 ? min(P.xw, P.wo - tile_x * P.xw) : min(P.n_valid, P.ptot - pix0);
    const int cpc = (n_lim + S - 1) / S;               // pixel rows one rank finishes
    const int jb = min(split * cpc, n_lim), je = min(jb + cpc, n_lim);
    // best-effort flavour: what this CTA saw at entry.  Nothing is loaded then; the cluster agrees at its first barrier.
    const bool abort0 = BE && s_flags[0] != 0;

    {
        const int m0 = tile_m * TC_BM;
        // ---------------- TMA producer, part 1: fill the ring (no waits) ----------------
        // Warp 0 refills the ring and warp 1 issues the multiplications as whole warps: control flow, addresses and
        // descriptors are warp-uniform (uniform registers), one elected lane executes each instruction.  As code of a
        // single thread every instruction had its operands moved into uniform registers first: 540 cycles per K block in
        // the multiplication loop, whatever the tile's width.
        const uint32_t tx = (uint32_t)P.load_bytes;
        const int first = nkb < NS ? nkb : NS;
        // filter tap and channel block of the next K block to refill, carried along (2^32 / 1 does not fit the magic: one
        // channel block per tap is a copy)
        int tap = P.cblocks == 1 ? kb_begin + first : (int)__umulhi((unsigned)(kb_begin + first), P.cb_magic);
        int cb = kb_begin + first - tap * P.cblocks;
        auto next_kb = [&]() {
            if (++cb == P.cblocks) { cb = 0; tap++; }
        };
        // weights: 32 channels of one tap for this tile's 128 output channels
        auto load_a = [&](int s) { tma_load_3d(base + s * stage_bytes, &P.tm_w, bar_full + 8 * s, cb * TC_BK, tap, m0); };
        auto load_b = [&](int s) {
            const uint32_t dst = base + s * stage_bytes + TC_A_BYTES;
            // the per-tap sub-lattice and offsets come from a host table
            if (P.spatial) {
                tma_load_3d(dst, &P.tm_x[P.tap_map[tap]], bar_full + 8 * s, cb * TC_BK, tile_x * P.xw + P.tap_qx[tap],
                            tile_y * P.rows + P.tap_qy[tap]);
            } else {
                tma_load_2d(dst, &P.tm_x[0], bar_full + 8 * s, cb * TC_BK, tile_n * P.n_valid);
            }
        };
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
                tma_load_3d(base + lane * stage_bytes, &P.tm_w, bar_full + 8 * lane, bc0, t, m0);
                if (P.spatial) {
                    bmap = &P.tm_x[P.tap_map[t]];
                    bc1 = tile_x * P.xw + P.tap_qx[t];
                    bc2 = tile_y * P.rows + P.tap_qy[t];
                }
            }
            asm volatile("griddepcontrol.wait;" ::: "memory");
            // Only now may the next kernel of the stream begin its prologue (set-up, weight loads).  Released
            // any earlier, a chain of these kernels runs ahead without bound and parks its blocks on every SM;
            // in this order at most two grids of a chain are resident and the other SM slots stay free for
            // best-effort kernels.  One thread per CTA executing the instruction counts for the CTA.
            asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            if (lane < first && !abort0) {
                const uint32_t bdst = base + lane * stage_bytes + TC_A_BYTES;
                if (P.spatial) tma_load_3d(bdst, bmap, bar_full + 8 * lane, bc0, bc1, bc2);
                else tma_load_2d(bdst, bmap, bar_full + 8 * lane, bc0, bc1);
            }
            __syncwarp();
            if (lane == 0) tc_stamp(P, 2);   // ring filled (loads issued)
        }
        __syncwarp();

        // epilogue parameters of this lane's 4 output channels: model constants, requested right after the first loads so
        // that their latency is long gone when the accumulator is ready
        const int cbase = lane * 4;
        const int co = m0 + cbase;
        const bool cvalid = co < P.co;
        float4 sc = make_float4(1.f, 1.f, 1.f, 1.f), sh = make_float4(0.f, 0.f, 0.f, 0.f);
        float4 b2 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (cvalid) {
            if (P.ep & TC_EP_GB) {
                sc = __ldg(reinterpret_cast<const float4*>(P.gamma + co));
                sh = __ldg(reinterpret_cast<const float4*>(P.beta + co));
            } else if (P.ep & TC_EP_BIAS) {
                sh = __ldg(reinterpret_cast<const float4*>(P.bias + co));
            }
            if (P.bias2 != nullptr) b2 = __ldg(reinterpret_cast<const float4*>(P.bias2 + co));
        }
        const float lo = (P.ep & TC_EP_RELU) ? 0.f : -__int_as_float(0x7f800000);
        const bool has_res = (P.ep & TC_EP_RES) != 0;
        const bool rnd = (P.ep & TC_EP_ROUND) != 0;
        const bool gelu = (P.ep & TC_EP_GELU) != 0;

        if (warp == 0) {
            // ---------------- TMA producer, part 2: refill stages as the MMAs release them ----------------
            // (stage index and phase parity are carried along: a division by the runtime ring depth per K block
            // is dozens of cycles on this critical path)
            bool ok = true;
            int s = first == NS ? 0 : first;      // first < NS only when nkb < NS, and then this loop does not run
            uint32_t par = 0;                      // parity of the "empty" phase awaited: ((i / NS) - 1) & 1
            int issued = abort0 ? 0 : first;       // K blocks whose loads are out
            bool stop = abort0;
            // A second look at the preempt flag, behind the dependency wait: a best-effort kernel queued behind a
            // running one is resident early (programmatic dependent launch) and made its entry poll long before its
            // predecessor finished, possibly before the flag went up.  Its first loads are out (their barriers were
            // armed for both operands, so the activation loads had to follow the weight loads); it issues no more, and
            // the MMA warp only waits for those to land.
            if (BE && !stop) stop = __any_sync(0xffffffffu, *reinterpret_cast<const volatile int*>(P.preempt_flag) != 0);
            for (int i = first; i < nkb && ok && !stop; i++) {
                // loop-head poll of the preempt flag (every 4th K block): the load is issued before the wait for a
                // free stage and looked at after it, so its latency hides behind the wait
                int f = 0;
                if (BE && (i & 3) == 0) f = *reinterpret_cast<const volatile int*>(P.preempt_flag);
                ok = mbar_wait_warp(bar_empty + 8 * s, par);
                if (!ok) break;
                if (BE && __any_sync(0xffffffffu, f != 0)) { stop = true; break; }
                if (elect_one()) {
                    mbar_expect_tx(bar_full + 8 * s, tx);
                    load_a(s);
                    load_b(s);
                }
                next_kb();
                issued++;
                if (++s == NS) { s = 0; par ^= 1u; }
            }
            if (BE && stop && lane == 0) {
                s_flags[2] = (uint32_t)issued;     // first how far the loads got, then the request to stop
                __threadfence_block();
                s_flags[0] = 1;
            }
            if (!ok && lane == 0) s_flags[1] = 1;
        } else if (warp == 1) {
            // ---------------- MMA issuer ----------------
            bool ok = true, halted = false;
            const uint32_t idesc = umma_idesc_tf32(P.n_mma);
#ifdef REEF_DEBUG_AIDS
            const bool tr = lane == 0 && P.trace != nullptr && blockIdx.x == 0 && blockIdx.y == 0;
#endif
            int s = 0;
            uint32_t par = 0;
            uint64_t da = umma_desc_sw128(base);
            for (int i = 0; i < nkb; i++) {
                if (BE) {
                    const int w = mbar_wait_abortable_warp(bar_full + 8 * s, par, &s_flags[0]);
                    if (w == 2) {
                        // The producer stopped.  Loads it had issued may still be in flight: they must have landed
                        // before this CTA leaves or reuses its shared memory, so their barriers are awaited (bounded)
                        // without multiplying.
                        __threadfence_block();
                        const int issued = __shfl_sync(0xffffffffu, (int)s_flags[2], 0);
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
#ifdef REEF_DEBUG_AIDS
                if (tr && i == 0) P.trace[4] = clock64();          // first K block landed
                if (tr && i == nkb - 1) P.trace[5] = clock64();    // last K block landed
#endif
                const uint64_t db = da + (uint64_t)(TC_A_BYTES >> 4);
                // one tcgen05.mma covers K = 8 tf32 = 32 bytes
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < TC_BK / 8; k++)
                        umma_tf32(tmem, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (i > 0 || k > 0) ? 1u : 0u);
                    if (i + NS < nkb) umma_commit(bar_empty + 8 * s);   // frees the stage, where it is refilled, once these MMAs have read it
                    if (i == nkb - 1) umma_commit(bar_acc);
                }
                __syncwarp();
                da += (uint64_t)(stage_bytes >> 4);
                if (++s == NS) { s = 0; par ^= 1u; da = umma_desc_sw128(base); }
            }
            // stopped early: the accumulator barrier completes when the multiplications issued so far have
            if (BE && halted && ok && elect_one()) umma_commit(bar_acc);
            __syncwarp();
            if (!ok && lane == 0) s_flags[1] = 1;
        }
        __syncwarp();
        if (warp != 0) asm volatile("griddepcontrol.wait;" ::: "memory");
        // the first two residual rows of this warp's pass over its pixel rows (rows jb + warp + 8u): requested now, used
        // after the exchange
        float4 rpre[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            rpre[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            const int jr = warp + 8 * u;
            if (has_res && cvalid && jr < je - jb)
                rpre[u] = ld_activation(P.res + (size_t)(pix0 + jb + jr) * P.co + co);
        }

        // ---------------- epilogue: all eight warps ----------------
        bool ok = mbar_wait(bar_acc, 0);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        __syncthreads();
        if (tid == 0) tc_stamp(P, 6);   // accumulator complete
        const bool my_abort = BE && s_flags[0] != 0;   // final: producer and MMA warp are past their loops
        if (!ok || s_flags[1]) {
            ok = false;
            if (tid == 0 && P.error_word) *reinterpret_cast<volatile int*>(P.error_word) = 1;
        }
        // Phase A — eight warps move the accumulator tile TMEM -> registers -> shared memory as stage[pixel][channel]
        // (warp w reads TMEM lanes 32*(w%4).., its hardware quadrant, and every other 16 columns, by w/4).  The stage ring
        // is free by now and is reused for this.
        // Phase B — the tile is finished pixel row by pixel row with 128-bit accesses: one warp per pixel, a lane owns 4
        // consecutive output channels.  With a K split, rank q finishes rows [q*cpc, (q+1)*cpc) and reads every rank's
        // partial of them from its shared memory; 128-bit remote loads, 16 in flight per lane, take half the time of a
        // bulk copy per peer into a receive area (1800 cycles from its issue to the owner's barrier).
        const int quad = warp & 3, half = warp >> 2;
        const int row = quad * 32 + lane;              // TMEM lane == output channel within the tile
        const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16);
        float* stage = reinterpret_cast<float*>(smem);
        if (ok && !my_abort) {
            for (int j0 = half * 16; j0 < n_lim; j0 += 64) {
                uint32_t r[32];
                tmem_ld16_nowait(taddr + j0, r);
                if (j0 + 32 < n_lim) tmem_ld16_nowait(taddr + j0 + 32, r + 16);
                tmem_ld_wait();
                float* dst = stage + j0 * TC_BM + row;
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (j0 + j < n_lim) dst[j * TC_BM] = __uint_as_float(r[j]);
                if (j0 + 32 < n_lim) {
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        if (j0 + 32 + j < n_lim) dst[(32 + j) * TC_BM] = __uint_as_float(r[16 + j]);
                }
            }
        }
        if (tid == 0) tc_stamp(P, 7);   // accumulator tile staged in shared memory
        // The accumulator is out of tensor memory once every warp has passed the barrier below, so the allocating
        // warp frees it there and not at the very end: nothing is then left to do between a CTA's last store and
        // its exit, which is what the next kernel of the stream waits for.
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        bool abort_all = my_abort;
        if (S > 1) {
            // cluster barrier #1: every rank's tile is staged.  (Nothing is written into a peer's shared memory, and a
            // peer's is not read before this barrier: only behind it is every CTA of the cluster known to have started.)
            cluster_sync_all();
            if (warp == 1) tmem_free(tmem, (uint32_t)P.tmem_cols);
            if (tid == 0) tc_stamp(P, 3);
            if (BE) {
                // every rank learns whether ANY rank of the cluster stopped for the preempt flag: one thread per rank
                // reads that rank's abort word through distributed shared memory; all ranks compute the same OR
                uint32_t f = 0;
                if (tid < S)
                    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(f) : "r"(mapa_shared(smem_u32((const void*)&s_flags[0]), (uint32_t)tid)) : "memory");
                abort_all = __syncthreads_or((int)f) != 0;
            }
        } else {
            __syncthreads();
            if (warp == 1) tmem_free(tmem, (uint32_t)P.tmem_cols);
        }
        if (tid == 0) tc_stamp(P, 8);
        if (ok && cvalid && !abort_all) {
            const uint32_t st = smem_u32(stage);
#define TC_FINISH(RB, SMAX)                                                                                                            \
    do {                                                                                                                               \
        if (gelu) tc_finish_rows<RB, SMAX, true>(P, st, S, jb, je, warp, cbase, co, pix0, sc, sh, lo, rnd, has_res, b2, rpre);         \
        else tc_finish_rows<RB, SMAX, false>(P, st, S, jb, je, warp, cbase, co, pix0, sc, sh, lo, rnd, has_res, b2, rpre);             \
    } while (0)
            if (S == 1) TC_FINISH(4, 1);
            else if (S == 2) TC_FINISH(4, 2);
            else if (S <= 4) TC_FINISH(4, 4);
            else TC_FINISH(2, TC_MAX_SPLITS);
#undef TC_FINISH
        }
        // cluster barrier #2: nobody reads a peer's shared memory any more, every CTA may exit
        if (S > 1) cluster_arrive_relaxed();
        if (S > 1) cluster_wait();      // barrier #2
        if (tid == 0) tc_stamp(P, 9);   // rows finished
        if (BE && abort_all && tid == 0 && P.stamps != nullptr) {
            // measurement only: when this block saw the preempt flag and left (device clock)
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            atomicMin(&P.stamps[0], t);
            atomicMax(&P.stamps[1], t);
        }
        if (P.task_slot != nullptr && ok && !abort_all) {
            __syncthreads();
            if (tid == 0) red_relaxed_gpu_add(P.task_slot, 1);
        }
    }

    if (tid == 32) tc_stamp(P, 10);   // leaving
}

}  // namespace reef
