// conv2d family in fp32: implicit GEMM, channels-last activations, OHWI weights.
//
//   out[y][x][co] = sum_{ky,kx,ci} in[y*sh+ky-ph][x*sw+kx-pw][ci] * W[co][ky][kx][ci]   (zero pad)
//   then (+residual[y][x][co]) (+bias[co] | *gamma[co]+beta[co]) (ReLU)
// (reference: resource/resnet152/resnet152.cu:315-363,3393-3418; args in, W, out, [residual], [bias | gamma, beta]).
//
// GEMM view: M = pixels (ho*wo), N = co, K = kh*kw*ci with ci fastest, so a K slice of 16 or 32 is one contiguous 64- or 128-byte run
// of both the activation pixel and the weight row.  The exact-fp32 path of the library: used for the 3-channel NCHW
// stem, odd shapes, and wherever the schedule asks for fp32 instead of TF32 tensor cores.
//
// What bounds it: 128 fp32 multiply-adds per clock and SM fed from shared memory at one word per lane and clock, so that
// CUDA cores reach their rate only on tiles of 8x8 outputs per thread — and at batch 1 there are far too few of those (a
// 13x13 layer of 256 channels is 12 tiles of 64x64, which left 136 SMs idle: 133 us; small tiles by fp32 instructions,
// 20 us).  The products therefore go to the tensor cores with exactly split operands (bf16_split.cuh, mma.sync m16n8k16).
// Accumulators are fp32: the large products are added up over 32 K positions and then to the running sum with a rounding
// addition (the tensor core truncates), the small ones in accumulators of their own.  Against fp64 the result is as close
// as a chain of fp32 fused multiply-adds, or closer.
//
// Work split: the eight warps of a block share one K loop.  A WARP computes a tile of 16 pixels x 32 or 16 channels over
// every KG-th K slice, KG = 1, 2, 4 or 8 warps sharing a tile and 8/KG tiles (neighbouring pixels) making a block.  Warps
// run on their own through a private ring of cp.async stages, no block barrier in the loop; the KG partial tiles meet in
// shared memory, summed in a fixed order.  A lane's K positions in a fragment are four consecutive ones (the order inside
// a slice is free as long as both operands agree), so an operand row is read with one 128-bit load.
// Measured, 3x3 256 -> 256 at 13x13: 133 -> 13.6 us; 3x3 512 -> 512 at 7x7: 261 -> 18.3 us; ResNet-50 at 193x193, a request:
// 3.39 -> 0.64 ms.
#pragma once
#include "bf16_split.cuh"
#include "task.cuh"

namespace reef {

constexpr int CBK = 16;                       // K slice
constexpr int CTP = 16;                       // pixels of a warp tile
constexpr int kConvSimtRing = 98304;          // eight warps' stages; two blocks fit an SM
constexpr int kConvSimtSmem = kConvSimtRing + 128;

// Channels of the warp tile and K groups of a shape: the least time by what was measured.  One block on an SM takes 0.57 us
// per slice of eight 16x32 tiles and 0.41 us of 16x16 (splitting operands into bf16 is most of it), blocks that share an SM
// overlap by a sixth; launch, prologue and epilogue take 3.5 us, every further block of an SM half a microsecond.
struct ConvSimtTile {
    int tc, kg;
};
__host__ inline ConvSimtTile conv_simt_tile(int ptot, int co, int ktot) {
    const int slices = (ktot + CBK - 1) / CBK;
    ConvSimtTile best = {32, 1};
    double best_t = 1e30;
    for (int tc = 32; tc >= 16; tc /= 2)
        for (int kg = 1; kg <= 8; kg *= 2) {
            const int tp = CTP * 8 / kg;
            const double blocks = (double)((ptot + tp - 1) / tp) * ((co + tc - 1) / tc);
            const int share = (int)((blocks + 147) / 148);
            const double t = 3.5 + 0.5 * share + (share > 1 ? 0.84 * share : 1.0) * ((slices + kg - 1) / kg) * (tc == 32 ? 0.566 : 0.41);
            if (t < best_t) {
                best_t = t;
                best = {tc, kg};
            }
        }
    return best;
}

// chunks of four channels in one tap each, and a bit per filter row and column
__host__ __device__ inline bool conv_simt_fast(const ConvP& p) {
    return !p.nchw && ((p.ci | p.ics | p.ioff) & 3) == 0 && p.kh <= 31 && p.kw <= 31;
}
// bit t: position first + t lies inside [0, n), for the t < taps <= 31
__device__ __forceinline__ int taps_inside(int first, int n, int taps) {
    const unsigned below = (1u << max(0, min(taps, n - first))) - 1u, before = (1u << max(0, min(31, -first))) - 1u;
    return (int)(below & ~before);
}

// 16 pixels x 8 NT channels per warp.  FAST: channels-last input whose 16-byte chunks lie in one tap each; else (planar
// input, odd channel counts) element by element.
template <int NT, int STAGES, bool FAST>
__device__ __forceinline__ bool conv_simt_tile_body(const KTask& t, int vb, float* ring, const int* flag) {
    constexpr int TP = CTP, TC = 8 * NT, CROW = CBK, STAGE = (TP + TC) * CROW;
    static_assert(8 * STAGES * STAGE * 4 <= kConvSimtRing && 8 * TP * (TC + 4) * 4 <= kConvSimtRing, "ring too small");
    const ConvP& p = t.p.conv;
    const float* __restrict__ in = (const float*)t.a[0];
    const float* __restrict__ wgt = (const float*)t.a[1];
    float* __restrict__ out = (float*)t.a[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int KG = p.kgroups, group = warp % KG;
    const int tile_c = vb % p.tiles_c, tile_p = vb / p.tiles_c;
    const int p0 = (tile_p * (8 / KG) + warp / KG) * TP, c0 = tile_c * TC;
    const int slices = (p.ktot + CBK - 1) / CBK;
    float* mine = ring + warp * STAGES * STAGE;
    const uint32_t mine_s = (uint32_t)__cvta_generic_to_shared(mine);

    // Loader: this lane copies chunk lane % 4 of rows lane / 4 + 8 i (four lanes read the 64 bytes of a row).  Per pixel
    // row the offset of its first tap, and the taps inside the image: FAST, one bit per filter row and column, else the
    // position of the first tap.  Rows beyond the last pixel repeat it (their results are not stored).
    const int lrow = lane >> 2, lk = (lane & 3) * 4;
    int off[TP / 8];
    int in_y[TP / 8], in_x[TP / 8];
#pragma unroll
    for (int i = 0; i < TP / 8; i++) {
        const int pix = min(p0 + lrow + 8 * i, p.ptot - 1);
        const int oy = pix / p.wo;
        const int iy = oy * p.sh - p.ph, ix = (pix - oy * p.wo) * p.sw - p.pw;
        off[i] = p.nchw ? iy * p.wi + ix : (iy * p.wi + ix) * p.ics + p.ioff;
        in_y[i] = FAST ? taps_inside(iy, p.hi, p.kh) : iy;
        in_x[i] = FAST ? taps_inside(ix, p.wi, p.kw) : ix;
    }
    const float* wrow = wgt + (size_t)(c0 + lrow) * p.ktot + lk;
    const int wlast = p.co - 1 - c0 - lrow, wstep = 8 * p.ktot;   // rows further than wlast are beyond the last channel
    // slice kt = group, group + KG, ...: tap and channel of this lane's chunk are carried along
    int kt = group, cb = group * CBK + lk, ky = 0, kx = 0;
    auto settle = [&]() {
        while (cb >= p.ci) {
            cb -= p.ci;
            if (++kx == p.kw) {
                kx = 0;
                ky++;
            }
        }
    };
    if (FAST) settle();
    auto load = [&](int stage) {
        const uint32_t a = mine_s + (uint32_t)(stage * STAGE + lrow * CROW + lk) * 4;
        const int k = kt * CBK;
        if (FAST) {
            const bool kin = k + lk < p.ktot;
            const int d = (ky * p.wi + kx) * p.ics + cb;
#pragma unroll
            for (int i = 0; i < TP / 8; i++) {
                const bool v = kin && (in_y[i] >> ky & in_x[i] >> kx & 1);
                const float* src = in + (v ? off[i] + d : 0);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a + i * 8 * CROW * 4), "l"(src), "r"(v ? 16 : 0) : "memory");
            }
            const float* src = wrow + k;
#pragma unroll
            for (int j = 0; j < TC / 8; j++, src += wstep)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a + (TP + j * 8) * CROW * 4), "l"(kin && 8 * j <= wlast ? src : wgt),
                             "r"(kin && 8 * j <= wlast ? 16 : 0)
                             : "memory");
            cb += KG * CBK;
            settle();
        } else {
#pragma unroll 1
            for (int e = 0; e < 4; e++) {
                const int ke = k + lk + e;
                const bool kin = ke < p.ktot;
                const int tp = ke / p.ci, c = ke - tp * p.ci;
                const int dy = tp / p.kw, dx = tp - dy * p.kw;
                const int d = p.nchw ? (c * p.hi + dy) * p.wi + dx : (dy * p.wi + dx) * p.ics + c;
#pragma unroll
                for (int i = 0; i < TP / 8; i++) {
                    const int iy = in_y[i] + dy, ix = in_x[i] + dx;
                    const bool v = kin && iy >= 0 && iy < p.hi && ix >= 0 && ix < p.wi;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(a + (i * 8 * CROW + e) * 4), "l"(in + (v ? off[i] + d : 0)), "r"(v ? 4 : 0) : "memory");
                }
                const float* src = wrow + k + e;
#pragma unroll
                for (int j = 0; j < TC / 8; j++, src += wstep)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(a + ((TP + j * 8) * CROW + e) * 4),
                                 "l"(kin && 8 * j <= wlast ? src : wgt), "r"(kin && 8 * j <= wlast ? 4 : 0)
                                 : "memory");
            }
        }
        kt += KG;
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };

    // D fragments: lane (g, c) = (lane / 4, lane % 4) holds pixels g and g + 8 of channels 2 c and 2 c + 1
    float sum[NT][4], big[NT][4], small[NT][4];
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) sum[j][e] = big[j][e] = small[j][e] = 0.f;
    const int g = lane >> 2, c = lane & 3;
    bool stopped = false;
    __syncthreads();                           // a persistent caller's previous tile is out of the ring
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++) {
        if (kt < slices) load(s);
        commit();
    }
    int stage = 0, fill = STAGES - 1, f = 0;
    for (int i0 = group, n = 0; i0 < slices; i0 += KG, n++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncwarp();                          // slice landed for every lane; the stage before it is free for every lane
        // best-effort flavour: loop-head poll of the preempt flag, every 8th slice of a warp, asked for four slices ahead
        if (flag != nullptr && (n & 7) == 3) f = ld_flag(flag);
        if (flag != nullptr && (n & 7) == 7 && __any_sync(0xffffffffu, f)) {
            stopped = true;
            break;
        }
        if (kt < slices) load(fill);
        commit();
        // (rows of 64 bytes without padding: the eight lanes of a 128-bit load's quarter read two rows = all 32 banks)
        const float* a = mine + stage * STAGE + g * CROW + c * 4;
        const float4 x0 = *reinterpret_cast<const float4*>(a), x1 = *reinterpret_cast<const float4*>(a + 8 * CROW);
        const Bf16Triple a0 = bf16_split(x0.x, x0.y), a1 = bf16_split(x1.x, x1.y), a2 = bf16_split(x0.z, x0.w), a3 = bf16_split(x1.z, x1.w);
#pragma unroll
        for (int j = 0; j < NT; j++) {
            const float4 w = *reinterpret_cast<const float4*>(a + (TP + 8 * j) * CROW);
            const Bf16Triple b0 = bf16_split(w.x, w.y), b1 = bf16_split(w.z, w.w);
            mma_bf16(small[j], a0.l, a1.l, a2.l, a3.l, b0.h, b1.h);
            mma_bf16(small[j], a0.h, a1.h, a2.h, a3.h, b0.l, b1.l);
            mma_bf16(small[j], a0.m, a1.m, a2.m, a3.m, b0.m, b1.m);
            mma_bf16(small[j], a0.m, a1.m, a2.m, a3.m, b0.h, b1.h);
            mma_bf16(small[j], a0.h, a1.h, a2.h, a3.h, b0.m, b1.m);
            mma_bf16(big[j], a0.h, a1.h, a2.h, a3.h, b0.h, b1.h);
        }
        if (n & 1) {
#pragma unroll
            for (int j = 0; j < NT; j++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    sum[j][e] += big[j][e];
                    big[j][e] = 0.f;
                }
        }
        if (++stage == STAGES) stage = 0;
        if (++fill == STAGES) fill = 0;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (__syncthreads_or(stopped)) return false;

    // partial tiles -> shared memory [warp][pixel][channel]
    constexpr int PROW = TC + 4;
    float* part = ring + warp * TP * PROW;
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
        for (int e = 0; e < 4; e += 2)
            *reinterpret_cast<float2*>(part + (g + 4 * e) * PROW + 8 * j + 2 * c) =
                make_float2(sum[j][e] + (big[j][e] + small[j][e]), sum[j][e + 1] + (big[j][e + 1] + small[j][e + 1]));
    __syncthreads();

    // epilogue: a thread finishes four channels of a pixel
    const float* res = (p.ep & EP_RES) ? (const float*)t.a[p.i_res] : nullptr;
    for (int item = tid; item < (8 / KG) * TP * (TC / 4); item += kThreads) {
        const int c4 = item % (TC / 4), row = item / (TC / 4);       // row: pixel within the block
        const int sub = row / TP, op = tile_p * (8 / KG) * TP + row, co = c0 + c4 * 4;
        if (op >= p.ptot || co >= p.co) continue;
        float4 sc = make_float4(1.f, 1.f, 1.f, 1.f), sh = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.ep & EP_GB) {
            sc = *reinterpret_cast<const float4*>((const float*)t.a[p.i_gamma] + co);
            sh = *reinterpret_cast<const float4*>((const float*)t.a[p.i_beta] + co);
        } else if (p.ep & EP_BIAS) {
            sh = *reinterpret_cast<const float4*>((const float*)t.a[p.i_bias] + co);
        }
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        if (res) r = *reinterpret_cast<const float4*>(res + (size_t)op * p.co + co);
        const float* src = ring + (size_t)(sub * KG * TP + row - sub * TP) * PROW + c4 * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int g = 0; g < KG; g++) {                               // fixed order: deterministic
            const float4 x = *reinterpret_cast<const float4*>(src + (size_t)g * TP * PROW);
            v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
        }
        if (split_sum_lost((v.x + v.y) + (v.z + v.w))) {
            // by fp32 multiply-adds over the taps inside the image (co is a multiple of four, p.co too)
            float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
            const int oy = op / p.wo, iy0 = oy * p.sh - p.ph, ix0 = (op - oy * p.wo) * p.sw - p.pw;
            const float* w = wgt + (size_t)co * p.ktot;
#pragma unroll 1
            for (int k = 0; k < p.ktot; k++, w++) {
                const int tap = k / p.ci, ch = k - tap * p.ci, ty = tap / p.kw;
                const int iy = iy0 + ty, ix = ix0 + tap - ty * p.kw;
                if (iy < 0 || iy >= p.hi || ix < 0 || ix >= p.wi) continue;
                const float x = in[p.nchw ? (ch * p.hi + iy) * p.wi + ix : (iy * p.wi + ix) * p.ics + p.ioff + ch];
                e.x = fmaf(x, w[0], e.x);
                e.y = fmaf(x, w[p.ktot], e.y);
                e.z = fmaf(x, w[2 * p.ktot], e.z);
                e.w = fmaf(x, w[3 * p.ktot], e.w);
            }
            if (split_sum_lost(v.x)) v.x = e.x;
            if (split_sum_lost(v.y)) v.y = e.y;
            if (split_sum_lost(v.z)) v.z = e.z;
            if (split_sum_lost(v.w)) v.w = e.w;
        }
        v.x += r.x; v.y += r.y; v.z += r.z; v.w += r.w;
        if (p.ep & EP_GB) {
            // explicit fused multiply-add: the three flavours of this body are compiled in different
            // kernels and must round identically
            v.x = fmaf(v.x, sc.x, sh.x); v.y = fmaf(v.y, sc.y, sh.y);
            v.z = fmaf(v.z, sc.z, sh.z); v.w = fmaf(v.w, sc.w, sh.w);
        } else {
            v.x += sh.x; v.y += sh.y; v.z += sh.z; v.w += sh.w;
        }
        if (p.ep & EP_GELU) {
            // exact-erf GELU (reference: resource/bert/bert.cu:167-173)
            v.x = v.x * (0.5f * erff(v.x * 0.70710678118654752440f) + 0.5f);
            v.y = v.y * (0.5f * erff(v.y * 0.70710678118654752440f) + 0.5f);
            v.z = v.z * (0.5f * erff(v.z * 0.70710678118654752440f) + 0.5f);
            v.w = v.w * (0.5f * erff(v.w * 0.70710678118654752440f) + 0.5f);
        }
        if (p.ep & EP_RELU) {
            v.x = fmaxf(v.x, 0.f); v.y = fmaxf(v.y, 0.f);
            v.z = fmaxf(v.z, 0.f); v.w = fmaxf(v.w, 0.f);
        }
        *reinterpret_cast<float4*>(out + (size_t)op * p.ocs + p.ooff + co) = v;
    }
    return true;
}

__device__ __forceinline__ bool body_conv_simt(const KTask& t, int vb, unsigned char* smem_raw, const int* flag) {
    float* ring = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
    const ConvP& p = t.p.conv;
    if (!conv_simt_fast(p)) return conv_simt_tile_body<4, 3, false>(t, vb, ring, flag);
    if (p.tile_c == 32) return conv_simt_tile_body<4, 4, true>(t, vb, ring, flag);
    return conv_simt_tile_body<2, 4, true>(t, vb, ring, flag);
}

}  // namespace reef
