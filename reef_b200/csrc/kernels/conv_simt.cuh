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
// What is left: a block alone on its SM keeps the tensor cores busy a quarter of the time, two of them half of it, and issue
// 82 % of what the schedulers can; so every instruction of a slice counts.  Addresses are worked out per tap instead of per slice,
// accumulators are not cleared, a remainder of the split is one multiply-add, and the set-up runs ahead of the wait for the previous
// kernel.  Measured, 3x3 256 -> 256 at 13x13: 133 us by fp32 instructions, 13.9 before these, 11.1 with them; 3x3 512 -> 512 at
// 7x7: 261, 19.6, 15.8.
#pragma once
#include <type_traits>

#include "bf16_split.cuh"
#include "task.cuh"

namespace reef {

constexpr int CBK = 16;                       // K slice
constexpr int CTP = 16;                       // pixels of a warp tile
constexpr int kConvSimtRing = 98304;          // eight warps' stages; two blocks fit an SM
constexpr int kConvSimtSmem = kConvSimtRing + 128;

// Channels of the warp tile and K groups of a shape: the least time by what was measured.  A slice of eight 16x32 tiles
// counts as 0.57 us for one block on an SM and one of 16x16 as 0.41 (the ratio decides; splitting operands into bf16 is most of it), blocks that share an SM
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
template <int NT, int STAGES, bool FAST, class Enter>
__device__ __forceinline__ bool conv_simt_tile_body(const KTask& t, int vb, float* ring, const int* flag, Enter enter) {
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
    // position of the first tap.  Rows beyond the last pixel or channel repeat the last one (their results are not stored).
    // What a slice needs beyond one address per row is worked out where the tap changes: with it done for every slice, and
    // the zeroing and adding of accumulators, a warp issued 358 instructions a slice, of which 156 multiply and split.
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
    unsigned woff[TC / 8];                     // rows of the weights, in elements from the block's first
#pragma unroll
    for (int j = 0; j < TC / 8; j++) woff[j] = (unsigned)(min(c0 + lrow + 8 * j, p.co - 1) - c0) * (unsigned)p.ktot;
    const int ktot = p.ktot, ci = p.ci, kstep = KG * CBK;
    // slice kt = group, group + KG, ...: tap and channel of this lane's chunk are carried along
    int k = group * CBK + lk, cb = k, ky = 0, kx = 0;
    const float* wslice = wgt + (size_t)c0 * ktot + k;
    int tap_off[TP / 8], tap_in[TP / 8];       // this lane's pixels under the current tap: offset, 16 (bytes) or 0 outside
    auto settle = [&](bool first) {
        if (!first && cb < ci) return;
        while (cb >= ci) {
            cb -= ci;
            if (++kx == p.kw) {
                kx = 0;
                ky++;
            }
        }
        const int d = (ky * p.wi + kx) * p.ics, y = min(ky, 31);   // (behind the last slice: no tap is bit 31)
#pragma unroll
        for (int i = 0; i < TP / 8; i++) {
            const bool v = in_y[i] >> y & in_x[i] >> kx & 1;
            tap_off[i] = v ? off[i] + d : 0;
            tap_in[i] = v ? 16 : 0;
        }
    };
    if (FAST) settle(true);
    auto load = [&](int stage) {
        const uint32_t a = mine_s + (uint32_t)(stage * STAGE + lrow * CROW + lk) * 4;
        if (FAST) {
            const bool kin = k < ktot;
#pragma unroll
            for (int i = 0; i < TP / 8; i++)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a + i * 8 * CROW * 4), "l"(in + tap_off[i] + cb), "r"(kin ? tap_in[i] : 0) : "memory");
            const float* src = kin ? wslice : wgt;
#pragma unroll
            for (int j = 0; j < TC / 8; j++)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a + (TP + j * 8) * CROW * 4), "l"(src + woff[j]), "r"(kin ? 16 : 0) : "memory");
            cb += kstep;
            settle(false);
        } else {
#pragma unroll 1
            for (int e = 0; e < 4; e++) {
                const int ke = k + e;
                const bool kin = ke < ktot;
                const int tp = ke / ci, c = ke - tp * ci;
                const int dy = tp / p.kw, dx = tp - dy * p.kw;
                const int d = p.nchw ? (c * p.hi + dy) * p.wi + dx : (dy * p.wi + dx) * p.ics + c;
#pragma unroll
                for (int i = 0; i < TP / 8; i++) {
                    const int iy = in_y[i] + dy, ix = in_x[i] + dx;
                    const bool v = kin && iy >= 0 && iy < p.hi && ix >= 0 && ix < p.wi;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(a + (i * 8 * CROW + e) * 4), "l"(in + (v ? off[i] + d : 0)), "r"(v ? 4 : 0) : "memory");
                }
                const float* src = kin ? wslice + e : wgt;
#pragma unroll
                for (int j = 0; j < TC / 8; j++)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(a + ((TP + j * 8) * CROW + e) * 4), "l"(src + woff[j]), "r"(kin ? 4 : 0) : "memory");
            }
        }
        k += kstep;
        wslice += kstep;
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
    if (!enter()) return false;
    __syncthreads();                           // a persistent caller's previous tile is out of the ring
    int loaded = group;                        // the slice that `load` fetches next
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++) {
        if (loaded < slices) load(s);
        loaded += KG;
        commit();
    }
    int stage = 0, fill = STAGES - 1, f = 0;
    auto turn = [&] {                          // the next slice has landed and the stage before it is free, for every lane
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncwarp();
    };
    auto refill = [&] {
        if (loaded < slices) load(fill);
        loaded += KG;
        commit();
        if (++fill == STAGES) fill = 0;
    };
    auto multiply = [&](auto even) {
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
            if (even.value) mma_bf16_zero(big[j], a0.h, a1.h, a2.h, a3.h, b0.h, b1.h);
            else mma_bf16(big[j], a0.h, a1.h, a2.h, a3.h, b0.h, b1.h);
        }
        if (++stage == STAGES) stage = 0;
    };
    // two slices at a time, whose large products are added up before they join the sum
    for (int i0 = group, n = 0; i0 < slices; i0 += 2 * KG, n++) {
        turn();
        refill();
        multiply(std::true_type());
        if (i0 + KG >= slices) break;
        turn();
        // best-effort flavour: loop-head poll of the preempt flag, every 8th slice of a warp, asked for four slices ahead
        if (flag != nullptr && (n & 3) == 1) f = ld_flag(flag);
        if (flag != nullptr && (n & 3) == 3 && __any_sync(0xffffffffu, f)) {
            stopped = true;
            break;
        }
        refill();
        multiply(std::false_type());
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) sum[j][e] += big[j][e];
    }
    if (slices <= group || ((slices - group + KG - 1) / KG & 1) == 0) {   // every slice's large products are in the sum
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) big[j][e] = 0.f;
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

template <class Enter>
__device__ __forceinline__ bool body_conv_simt(const KTask& t, int vb, unsigned char* smem_raw, const int* flag, Enter enter) {
    float* ring = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
    const ConvP& p = t.p.conv;
    if (!conv_simt_fast(p)) return conv_simt_tile_body<4, 3, false>(t, vb, ring, flag, enter);
    if (p.tile_c == 32) return conv_simt_tile_body<4, 4, true>(t, vb, ring, flag, enter);
    return conv_simt_tile_body<2, 4, true>(t, vb, ring, flag, enter);
}

}  // namespace reef
