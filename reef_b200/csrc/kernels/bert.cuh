// BERT families: embedding gather, LayerNorm (with optional residual add) and multi-head attention.
// The reference's TVM build spreads these over dozens of small kernels per layer — four softmax passes
// through an HBM scratch buffer, five LayerNorm launches, head split/merge transposes, a Q/sqrt(d) divide
// (reference: resource/bert/bert.cu:3-12,159-204,273-395).  Here each is one kernel; the dense projections
// run on the tensor-core GEMM with bias / GELU / residual fused in its epilogue (conv_tc.cuh).
#pragma once
#include "bf16_split.cuh"
#include "simple.cuh"

namespace reef {

// ---- embedding: out[s][h] = word[clamp(ids[s], 0, vocab-1)][h] + pos[s][h]  (reference: bert.cu:313-325) -----
// args: out, word_emb, ids (int64), pos_emb.  One thread = 4 channels of one token.
__device__ __forceinline__ bool body_embedding(const KTask& t, int vb, unsigned char*, const int*) {
    const int s = t.p.raw[0], h = t.p.raw[1], vocab = t.p.raw[2];
    float* out = (float*)t.a[0];
    const float* word = (const float*)t.a[1];
    const long long* ids = (const long long*)t.a[2];
    const float* pos = (const float*)t.a[3];
    const int h4 = h >> 2, total = s * h4;
#pragma unroll
    for (int it = 0; it < 4; it++) {
        const int i = vb * (kThreads * 4) + it * kThreads + threadIdx.x;
        if (i >= total) break;
        const int tok = i / h4, c = (i - tok * h4) << 2;
        long long id = ids[tok];
        id = id < 0 ? 0 : (id > vocab - 1 ? vocab - 1 : id);
        const float4 w = *reinterpret_cast<const float4*>(word + (size_t)id * h + c);
        const float4 p = *reinterpret_cast<const float4*>(pos + (size_t)tok * h + c);
        *reinterpret_cast<float4*>(out + (size_t)tok * h + c) = make_float4(w.x + p.x, w.y + p.y, w.z + p.z, w.w + p.w);
    }
    return true;
}

// ---- LayerNorm of x (+ residual): mean, two-pass variance, (x-mu)/sqrt(var+1e-12)*gamma+beta ------------------
// (reference: bert.cu:175-204,338-342,352-379; eps at :201).  args: out, x, [residual], gamma, beta.
// A row lives in registers, at most two 128-bit values a lane (h <= 1024, h % 128 == 0): one, two or four warps share a row, so that
// many SMs take part and every load of a launch is in flight at once.  What bounds a launch is its latency: the hand-over, one trip
// to L2 and two reductions.  A warp to a row of 768 kept its 12 to 24 loads in a chain of branches and eight rows on an SM:
// 128 rows 3.49 -> 1.86 us, 384 rows 3.59 -> 2.06 us a launch.
__host__ __device__ inline int ln_warps_per_row(int h) { return h <= 256 ? 1 : h <= 512 ? 2 : 4; }
constexpr int kLnRowsPerBlock = 8;   // with one warp to a row; schedules of earlier versions have it for every width
// gamma and beta are model constants: they are asked into L2 before the wait for the previous kernel.  A model's weights have
// flushed them out since its last pass, and behind the reductions their trip from HBM would stand on the critical path
// (0.5 us a launch of 128 rows).
__device__ __forceinline__ void prefetch_layernorm(const KTask& t) {
    const int h = t.p.raw[1], first = t.p.raw[2] ? 3 : 2, lines = h >> 5;
    if ((int)threadIdx.x < 2 * lines) {
        const bool second = (int)threadIdx.x >= lines;
        const float* p = (const float*)t.a[first + (second ? 1 : 0)] + ((int)threadIdx.x - (second ? lines : 0)) * 32;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
    }
}
__device__ __forceinline__ bool body_layernorm(const KTask& t, int vb, unsigned char*, const int*) {
    __shared__ float sums[2][8];
    const int rows = t.p.raw[0], h = t.p.raw[1], has_res = t.p.raw[2], rows_per_block = t.p.raw[3];
    float* out = (float*)t.a[0];
    const float* x = (const float*)t.a[1];
    const float* res = has_res ? (const float*)t.a[2] : nullptr;
    const float* gamma = (const float*)t.a[has_res ? 3 : 2];
    const float* beta = (const float*)t.a[has_res ? 4 : 3];
    const int W = ln_warps_per_row(h), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int part = warp & (W - 1), sub = warp / W;          // this warp's share of its row, its row among the block's
    // the sum over a row: its warps' sums in their order
    auto row_sum = [&](float v, float* s) {
        v = warp_sum(v);
        if (W == 1) return v;
        if (lane == 0) s[warp] = v;
        __syncthreads();
        float all = s[sub * W];
        for (int q = 1; q < W; q++) all += s[sub * W + q];
        return all;
    };
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    int c[2];
    bool in[2];
    float4 g[2], b[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
        c[i] = ((i * W + part) * 32 + lane) * 4;
        in[i] = c[i] < h;
        g[i] = in[i] ? *reinterpret_cast<const float4*>(gamma + c[i]) : zero;
        b[i] = in[i] ? *reinterpret_cast<const float4*>(beta + c[i]) : zero;
    }
    __syncthreads();                           // a persistent caller's previous block is out of the sums
    for (int r0 = 0; r0 < rows_per_block; r0 += 8 / W) {
        const int row = vb * rows_per_block + r0 + sub;
        const size_t at = (size_t)row * h;
        float4 v[2], r[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const bool there = in[i] && row < rows;
            v[i] = there ? *reinterpret_cast<const float4*>(x + at + c[i]) : zero;
            r[i] = there && res ? *reinterpret_cast<const float4*>(res + at + c[i]) : zero;
        }
        float sum = 0.f, sq = 0.f;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            v[i].x += r[i].x; v[i].y += r[i].y; v[i].z += r[i].z; v[i].w += r[i].w;
            sum += (v[i].x + v[i].y) + (v[i].z + v[i].w);
        }
        const float mu = row_sum(sum, sums[0]) / (float)h;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            v[i].x -= mu; v[i].y -= mu; v[i].z -= mu; v[i].w -= mu;
            if (in[i]) sq += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
        }
        const float rstd = 1.0f / sqrtf(row_sum(sq, sums[1]) / (float)h + 1e-12f);
#pragma unroll
        for (int i = 0; i < 2; i++)
            if (in[i] && row < rows)
                *reinterpret_cast<float4*>(out + at + c[i]) = make_float4(v[i].x * rstd * g[i].x + b[i].x, v[i].y * rstd * g[i].y + b[i].y,
                                                                          v[i].z * rstd * g[i].z + b[i].z, v[i].w * rstd * g[i].w + b[i].w);
    }
    return true;
}

// ---- multi-head self-attention on a fused [S][3H] buffer (Q | K | V, head-major inside each H) ----------------
// scores = Q K^T / sqrt(d); mask[j] == 0 -> -inf; row softmax (max-subtracted, online over key chunks);
// ctx = P V   (reference: bert.cu:22-157 batch_matmul_4/5, :289-311 divide + transposes, :381-387 where,
// softmax :3-12,159-165,327-336,389-395).  args: qkv, [mask], out.  d == 64.
// fp32 throughout: both products run on the tensor cores with exactly split operands (bf16_split.cuh), every 16 positions
// of a sum added to the fp32 result with rounding.  One logical block = one head x 16 query rows; its eight warps divide
// the keys (a range of whole 16s each) and keep their own running maximum, sum and context, merged at the end in warp
// order.  A lane's four K positions are consecutive dimensions in the first product; in the second it holds eight
// consecutive dimensions of four keys, which are its columns of all eight 8-column tiles at once: operands are read with
// 128-bit loads either way.  The query fragments are split once per block.
//
// Two forms.  What bounds a pass that fits the SMs at once (up to 148 blocks) is its latency: keys and values go from L2
// straight into registers (250 of them, one block per SM), the next loads travelling during either product.  Beyond that
// what counts is how many warps hide the chains of dependent multiplications behind each other (2 us per 16 keys with one
// block on an SM): keys and values are staged through shared memory by cp.async and two blocks share an SM.
// Measured, 12 heads: 128 tokens 8.6 us by fp32 instructions, 7.8 in TF32 on tcgen05, 5.1 here; 384 tokens 30.9 and 14.4 us; error against fp64 0.3-0.5 of the fp32 instructions'.
constexpr int kAttChunk = 16;                              // keys a warp takes at a time
constexpr int kAttD = 64;
constexpr int kAttRowStride = kAttD + 4;
constexpr int kAttRows = 16;
constexpr int kAttMergeBytes = 8 * kAttRows * kAttRowStride * 4;        // contexts of the eight warps
constexpr int kAttStageBytes = 8 * 3 * kAttChunk * kAttD * 4;           // per warp two key buffers and one of values
constexpr int kAttFixedBytes = 4 * 3 * 32 * 16 + 2 * 8 * kAttRows * 4;  // query fragments, maxima and sums
__host__ inline bool att_staged(int s, int heads) { return heads * ((s + kAttRows - 1) / kAttRows) > 148; }
__host__ inline int att_smem(bool staged) { return kAttFixedBytes + (staged ? kAttStageBytes : kAttMergeBytes); }   // 103 / 41 KB
// 16-byte chunks of a staged row of keys / values are exchanged so that the eight lanes of a 128-bit load's quarter (two
// rows x four chunks of keys; four rows x two chunks of values) meet different banks
__device__ __forceinline__ int att_swz_k(int row) { return (row & 1) << 2; }
__device__ __forceinline__ int att_swz_v(int row) { return ((row >> 1) & 1) | (((row >> 2) & 1) << 2); }
template <bool STAGED>
__device__ __forceinline__ bool attention_rows(const KTask& t, int vb, unsigned char* smem_raw, const int* flag) {
    constexpr int ROWS = kAttRows;
    const int S = t.p.raw[0], heads = t.p.raw[1], has_mask = t.p.raw[3];
    const int H = heads * kAttD;
    const float* qkv = (const float*)t.a[0];
    const float* mask = has_mask ? (const float*)t.a[1] : nullptr;
    float* out = (float*)t.a[has_mask ? 2 : 1];
    uint4* Qs = reinterpret_cast<uint4*>(smem_raw);                       // [k step][h, m, l][lane]: A fragments
    float* ml = reinterpret_cast<float*>(Qs + 4 * 3 * 32);                // [warp][row]: maximum, then [warp][row]: sum
    float* part = ml + 2 * 8 * ROWS;                                      // [warp][row][dimension], over the stages
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const int rblocks = (S + ROWS - 1) / ROWS;
    const int head = vb / rblocks, row0 = (vb - head * rblocks) * ROWS;
    const float scale = 0.125f;                                           // 1 / sqrt(64)
    const float ninf = -__int_as_float(0x7f800000);
    const float* base = qkv + head * kAttD;
    __syncthreads();                           // a persistent caller's previous block is out of shared memory
    if (warp < 4) {
        const int ks = warp, row = row0 + g;
        const float4 x = *reinterpret_cast<const float4*>(base + (size_t)min(row, S - 1) * 3 * H + ks * 16 + c * 4);
        const float4 y = *reinterpret_cast<const float4*>(base + (size_t)min(row + 8, S - 1) * 3 * H + ks * 16 + c * 4);
        const Bf16Triple a0 = bf16_split(x.x, x.y), a1 = bf16_split(y.x, y.y), a2 = bf16_split(x.z, x.w), a3 = bf16_split(y.z, y.w);
        Qs[(warp * 3 + 0) * 32 + lane] = make_uint4(a0.h, a1.h, a2.h, a3.h);
        Qs[(warp * 3 + 1) * 32 + lane] = make_uint4(a0.m, a1.m, a2.m, a3.m);
        Qs[(warp * 3 + 2) * 32 + lane] = make_uint4(a0.l, a1.l, a2.l, a3.l);
    }
    __syncthreads();

    const int range = ((S + 7) / 8 + 15) / 16 * 16;
    const int k_begin = warp * range, k_end = min(S, k_begin + range);
    float m[2] = {ninf, ninf}, l[2] = {0.f, 0.f}, ctx[8][4];
#pragma unroll
    for (int j = 0; j < 8; j++) ctx[j][0] = ctx[j][1] = ctx[j][2] = ctx[j][3] = 0.f;
    // keys k0 .. k0 + 15 of K: tile j, k step ks; of V: keys 2 c, 2 c + 1, 2 c + 8, 2 c + 9, dimensions 8 g .. 8 g + 7 (keys
    // beyond the sequence repeat the last one: their probability is zero)
    float4 kf[2][4];
    float vf[4][8];
    auto load_k = [&](int k0) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const float* src = base + (size_t)min(k0 + 8 * j + g, S - 1) * 3 * H + H + c * 4;
#pragma unroll
            for (int ks = 0; ks < 4; ks++) kf[j][ks] = *reinterpret_cast<const float4*>(src + ks * 16);
        }
    };
    // staged form: K buffers 0 and 1, V buffer, 16 rows of 256 bytes each
    float* mine = part + warp * 3 * kAttChunk * kAttD;
    const uint32_t mine_s = (uint32_t)__cvta_generic_to_shared(mine);
    auto stage = [&](int k0, int which, uint32_t dst, bool values) {   // which: 1 keys, 2 values of the token row
        if (k0 < k_end) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int row = 2 * i + (lane >> 4), chunk = lane & 15;
                const float* src = base + (size_t)min(k0 + row, S - 1) * 3 * H + which * H + chunk * 4;
                const uint32_t d = dst + row * 256 + ((chunk ^ (values ? att_swz_v(row) : att_swz_k(row))) << 4);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    bool stopped = false;
    if (STAGED) {
        stage(k_begin, 1, mine_s, false);
        stage(k_begin, 2, mine_s + 8192, true);
    } else if (k_begin < k_end) {
        load_k(k_begin);
    }
    int buf = 0, f = flag != nullptr ? ld_flag(flag) : 0;
#pragma unroll 1
    for (int k0 = k_begin; k0 < k_end; k0 += kAttChunk) {
        // best-effort flavour: loop-head poll of the preempt flag, asked for a step ahead
        if (flag != nullptr && k0 > k_begin) {
            if (__any_sync(0xffffffffu, f)) {
                stopped = true;
                break;
            }
            f = ld_flag(flag);
        }
        if (STAGED) {
            stage(k0 + kAttChunk, 1, mine_s + (buf ^ 1) * 4096, false);
            asm volatile("cp.async.wait_group 2;" ::: "memory");       // this step's keys (behind them: values, next keys)
            __syncwarp();
        } else {
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const float* src = base + (size_t)min(k0 + 2 * c + (u & 1) + 8 * (u >> 1), S - 1) * 3 * H + 2 * H + 8 * g;
                *reinterpret_cast<float4*>(&vf[u][0]) = *reinterpret_cast<const float4*>(src);
                *reinterpret_cast<float4*>(&vf[u][4]) = *reinterpret_cast<const float4*>(src + 4);
            }
        }
        // ---- scores; s[j][e]: row g + 8 (e / 2), key k0 + 8 j + 2 c + e % 2 ----
        float s[2][4];
#pragma unroll
        for (int j = 0; j < 2; j++) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < 4; ks++) {
            if (STAGED) {
#pragma unroll
                for (int j = 0; j < 2; j++)
                    kf[j][ks] = *reinterpret_cast<const float4*>(mine + buf * 1024 + (8 * j + g) * 64 + ((4 * ks + c) ^ att_swz_k(g)) * 4);
            }
            const Bf16Triple b0[2] = {bf16_split(kf[0][ks].x, kf[0][ks].y), bf16_split(kf[1][ks].x, kf[1][ks].y)};
            const Bf16Triple b1[2] = {bf16_split(kf[0][ks].z, kf[0][ks].w), bf16_split(kf[1][ks].z, kf[1][ks].w)};
            const uint4 qh = Qs[(ks * 3 + 0) * 32 + lane], qm = Qs[(ks * 3 + 1) * 32 + lane], ql = Qs[(ks * 3 + 2) * 32 + lane];
            const Bf16Triple a[4] = {{qh.x, qm.x, ql.x}, {qh.y, qm.y, ql.y}, {qh.z, qm.z, ql.z}, {qh.w, qm.w, ql.w}};
            float d[2][4];
            mma_split(d, a, b0, b1);
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int e = 0; e < 4; e++) s[j][e] += d[j][e];
        }
        if (!STAGED) load_k(k0 + kAttChunk);
        // ---- mask, running maximum, probabilities ----
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int key = k0 + 8 * j + 2 * c + e;
                const bool dead = key >= k_end || (mask && mask[key] == 0.f);
                s[j][e] = dead ? ninf : s[j][e] * scale;
                s[j][2 + e] = dead ? ninf : s[j][2 + e] * scale;
            }
#pragma unroll
        for (int r = 0; r < 2; r++) {
            float top = fmaxf(fmaxf(s[0][2 * r], s[0][2 * r + 1]), fmaxf(s[1][2 * r], s[1][2 * r + 1]));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            const float mnew = fmaxf(m[r], top);
            float add = 0.f;
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int e = 2 * r; e < 2 * r + 2; e++) {
                    s[j][e] = s[j][e] == ninf ? 0.f : expf(s[j][e] - mnew);
                    add += s[j][e];
                }
            if (k0 > k_begin) {   // (the first step has nothing to rescale)
                const float corr = mnew == ninf ? 1.f : expf(m[r] - mnew);
                l[r] = l[r] * corr + add;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    ctx[j][2 * r] *= corr;
                    ctx[j][2 * r + 1] *= corr;
                }
            } else {
                l[r] = add;
            }
            m[r] = mnew;
        }
        Bf16Triple p[4];
#pragma unroll
        for (int q = 0; q < 4; q++) p[q] = bf16_split(s[q >> 1][2 * (q & 1)], s[q >> 1][2 * (q & 1) + 1]);
        // ---- context: column g of tile j = dimension 8 g + j ----
        if (STAGED) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");       // this step's values
            __syncwarp();
        }
#pragma unroll
        for (int j0 = 0; j0 < 8; j0 += 4) {
            if (STAGED) {
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int row = 2 * c + (u & 1) + 8 * (u >> 1);
                    *reinterpret_cast<float4*>(&vf[u][j0]) = *reinterpret_cast<const float4*>(mine + 2048 + row * 64 + ((2 * g + j0 / 4) ^ att_swz_v(row)) * 4);
                }
            }
            Bf16Triple b0[4], b1[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                b0[j] = bf16_split(vf[0][j0 + j], vf[1][j0 + j]);
                b1[j] = bf16_split(vf[2][j0 + j], vf[3][j0 + j]);
            }
            float d[4][4];
            mma_split(d, p, b0, b1);
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int e = 0; e < 4; e++) ctx[j0 + j][e] += d[j][e];
        }
        if (STAGED) {
            __syncwarp();                                               // every lane has read this step's values
            stage(k0 + kAttChunk, 2, mine_s + 8192, true);
            buf ^= 1;
        }
    }
    if (STAGED) asm volatile("cp.async.wait_all;" ::: "memory");
    if (__syncthreads_or(stopped)) return false;

    // ---- the eight warps' parts meet: lane (g, c) holds dimensions 16 c .. 16 c + 15 of its rows ----
#pragma unroll
    for (int r = 0; r < 2; r++) {
        float sum = l[r];
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        const int row = g + 8 * r;
        if (c == 0) {
            ml[warp * ROWS + row] = m[r];
            ml[(8 + warp) * ROWS + row] = sum;
        }
        float* dst = part + (warp * ROWS + row) * kAttRowStride + 16 * c;
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int q = 0; q < 2; q++)
                *reinterpret_cast<float4*>(dst + 8 * h + 4 * q) =
                    make_float4(ctx[4 * q][2 * r + h], ctx[4 * q + 1][2 * r + h], ctx[4 * q + 2][2 * r + h], ctx[4 * q + 3][2 * r + h]);
    }
    __syncthreads();
    // sixteen lanes share a row: each works out the factor of one warp's part, the others have it from there
    const int row = threadIdx.x >> 4, d0 = (threadIdx.x & 15) * 4;
    const float mw = ml[(lane & 7) * ROWS + row];
    float top = mw;
#pragma unroll
    for (int q = 1; q < 8; q <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, q));
    const float fw = mw == ninf ? 0.f : expf(mw - top);
    float sum = 0.f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < 8; w++) {          // fixed order: deterministic
        const float f = __shfl_sync(0xffffffffu, fw, (lane & 16) + w);
        sum = fmaf(f, ml[(8 + w) * ROWS + row], sum);
        const float4 x = *reinterpret_cast<const float4*>(part + (w * ROWS + row) * kAttRowStride + d0);
        o.x = fmaf(f, x.x, o.x); o.y = fmaf(f, x.y, o.y); o.z = fmaf(f, x.z, o.z); o.w = fmaf(f, x.w, o.w);
    }
    if (row0 + row < S) {
        const float inv = 1.0f / sum;
        o.x *= inv; o.y *= inv; o.z *= inv; o.w *= inv;
        if (split_sum_lost((o.x + o.y) + (o.z + o.w))) {
            // by fp32 multiply-adds: the row's largest score, then its probabilities and their sum over the values
            const float* q = base + (size_t)(row0 + row) * 3 * H;
            float high = ninf, total = 0.f;
            float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
            for (int pass = 0; pass < 2; pass++)
#pragma unroll 1
                for (int key = 0; key < S; key++) {
                    const float* kv = base + (size_t)key * 3 * H + H;
                    float sc = 0.f;
#pragma unroll 1
                    for (int i = 0; i < kAttD; i++) sc = fmaf(q[i], kv[i], sc);
                    sc = mask && mask[key] == 0.f ? ninf : sc * scale;
                    if (pass == 0) {
                        high = fmaxf(high, sc);
                        continue;
                    }
                    const float pr = sc == ninf ? 0.f : expf(sc - high);
                    const float4 v = *reinterpret_cast<const float4*>(kv + H + d0);
                    total += pr;
                    e.x = fmaf(pr, v.x, e.x); e.y = fmaf(pr, v.y, e.y); e.z = fmaf(pr, v.z, e.z); e.w = fmaf(pr, v.w, e.w);
                }
            const float by = 1.0f / total;
            if (split_sum_lost(o.x)) o.x = e.x * by;
            if (split_sum_lost(o.y)) o.y = e.y * by;
            if (split_sum_lost(o.z)) o.z = e.z * by;
            if (split_sum_lost(o.w)) o.w = e.w * by;
        }
        *reinterpret_cast<float4*>(out + (size_t)(row0 + row) * H + head * kAttD + d0) = o;
    }
    return true;
}

}  // namespace reef
