// Host side of the tcgen05 convolution: tile/split planning, TMA tensor maps, cluster launch.
#include "conv_tc.cuh"

#include <cmath>
#include <cstdlib>
#include <cstring>
#include <string>

#include "registry.h"

namespace reef {

static int ceil_div_i(int a, int b) { return (a + b - 1) / b; }

// ---- planning (needs no GPU) --------------------------------------------------------------------
// One candidate plan: pixel tiles of at most `cap` pixels, K split over `want` ranks (0: the default of a name that fixes
// only its tile cap).
static int tc_plan_cap(const ConvP& p, int cap, int want, TcPlan* pl) {
    memset(pl, 0, sizeof(*pl));
    pl->spatial = (p.kh * p.kw > 1 || p.sh > 1 || p.ph || p.pw) ? 1 : 0;
    pl->xsplit = 1;
    pl->xw = p.wo;
    if (pl->spatial && p.wo > cap) {
        // rows wider than a tile: every row is cut into pieces of about the same width, the last one ragged
        pl->xw = ceil_div_i(p.wo, ceil_div_i(p.wo, cap));
        if (pl->xw < 8) return REEF_NOT_FOUND;
        pl->xsplit = ceil_div_i(p.wo, pl->xw);
        pl->rows = 1;
        pl->n_valid = pl->xw;
        pl->n_tiles = p.ho * pl->xsplit;
    } else if (pl->spatial) {
        int best = 1;
        const int rmax = cap / p.wo;
        const int lim = rmax < p.ho ? rmax : p.ho;
        for (int r = 1; r <= lim; r++)
            if (p.ho % r == 0) best = r;               // largest divisor of Ho that fits the tile
        if (best * 2 <= lim) best = ceil_div_i(p.ho, ceil_div_i(p.ho, lim));   // no useful divisor: ragged last tile
        pl->rows = best;
        pl->n_valid = best * p.wo;
        pl->n_tiles = ceil_div_i(p.ho, best);
    } else {
        int t = ceil_div_i(p.ptot, cap);
        pl->n_valid = ceil_div_i(p.ptot, t);
        pl->rows = 0;
        pl->n_tiles = ceil_div_i(p.ptot, pl->n_valid);
    }
    pl->n_mma = ceil_div_i(pl->n_valid, 16) * 16;
    if (pl->n_mma < 16) pl->n_mma = 16;
    pl->tmem_cols = 32;
    while (pl->tmem_cols < pl->n_mma) pl->tmem_cols *= 2;
    pl->m_tiles = ceil_div_i(p.co, TC_BM);
    pl->cblocks = ceil_div_i(p.ci, TC_BK);   // a ragged last channel block reads zeros beyond Cin (TMA out-of-bounds fill)
    pl->kb_total = p.kh * p.kw * pl->cblocks;
    // default: split K over a cluster until about 128 CTAs are in flight, keeping >= 2 K blocks per CTA
    const int base = pl->m_tiles * pl->n_tiles;
    int s = 1;
    if (want > 0) {
        while (s < want && s < TC_MAX_SPLITS && pl->kb_total >= s * 2) s *= 2;
    } else {
        while (s < TC_MAX_SPLITS && base * s * 2 <= 128 && pl->kb_total >= 2 * (s * 2)) s *= 2;
    }
    // every rank must own at least one K block and the cluster size stays a power of two
    for (;; s /= 2) {
        pl->kb_per_split = ceil_div_i(pl->kb_total, s);
        pl->splits = ceil_div_i(pl->kb_total, pl->kb_per_split);
        if (pl->splits == s || s == 1) break;
    }
    pl->b_bytes = pl->n_valid * 128;
    // Shared memory: at most TC_SMEM_CAP per CTA, so that two CTAs fit one SM (a real-time kernel beside the
    // early-launched prologue of its successor, or beside a best-effort kernel).  The stage ring is reused by
    // the epilogue for the staged accumulator tile (one 512-byte row per pixel) and, with a K split, the
    // exchange area recv[S-1][cpc_max][128].  Both are the chain kernel's (conv_tc_chain.cuh); the launches of one layer
    // stage nothing and have a receive area of their own (tc_place_recv).  They count for both all the same: a chain
    // gives its layers' results bit for bit, so a layer has one plan, and it must fit either kernel.
    const int budget = TC_SMEM_CAP - 1024 - 256;   // alignment slack and control words
    const int stage_bytes = TC_A_BYTES + pl->n_mma * 128;
    pl->stages = pl->kb_per_split < TC_MAX_STAGES ? pl->kb_per_split : TC_MAX_STAGES;
    while (pl->stages > 1 && pl->stages * stage_bytes > budget) pl->stages--;
    if (pl->stages * stage_bytes > budget || (pl->stages < 2 && pl->kb_per_split > 1)) return REEF_NOT_FOUND;
    int ring = pl->stages * stage_bytes;
    pl->cpc_max = ceil_div_i(pl->n_valid, pl->splits);
    pl->recv_offset_floats = pl->n_valid * TC_BM;
    const int epi = pl->n_valid * 512 + (pl->splits > 1 ? (pl->splits - 1) * pl->cpc_max * 512 : 0);
    if (epi > budget) return REEF_NOT_FOUND;
    pl->region_bytes = ring > epi ? ring : epi;
    pl->region_bytes = ((pl->region_bytes + 127) / 128) * 128;
    pl->smem = 1024 + pl->region_bytes + 256;   // alignment slack + data region + control words
    return REEF_SUCC;
}

// Where a plan's receive area goes (see TcParams::recv_offset).  Apart from the ring the peers may store into it at any time, over
// the ring only behind a cluster barrier that stands between the accumulator and the exchange (0.25 us): apart wherever shared
// memory has room for both, if need be with a stage less (3x3, 256 channels, 14x14: 4.5 us over five stages, 4.3 apart from four).
// `earlier`: no more shared memory than the plan took when partials were read from the peers' staging tiles; schedules written
// then state that size, and load with it.
static int tc_place_recv(TcPlan* pl, bool earlier) {
    const int budget = earlier ? pl->region_bytes : TC_SMEM_CAP - 1024 - 256;
    const int stage_bytes = TC_A_BYTES + pl->n_mma * 128;
    int ring = pl->stages * stage_bytes;
    pl->gpc = ceil_div_i(ceil_div_i(pl->n_valid, 4), pl->splits);
    const int recv = pl->splits > 1 ? pl->splits * pl->gpc * TC_BM * 16 : 0;
    if (recv > budget) return REEF_NOT_FOUND;
    if (!earlier && ring + recv > budget && pl->stages > 2 && ring - stage_bytes + recv <= budget) {
        pl->stages--;
        ring -= stage_bytes;
    }
    pl->recv_late = ring + recv > budget;
    pl->recv_offset = pl->recv_late ? 0 : ring;
    if (pl->recv_offset + recv > pl->region_bytes) pl->region_bytes = (pl->recv_offset + recv + 127) / 128 * 128;
    pl->smem = 1024 + pl->region_bytes + 256;
    return REEF_SUCC;
}

// Estimated SM cycles of one launch under a placed plan, up to a constant.  A batch-1 layer is a short chain of latencies beside
// a load stream, so neither the fewest bytes nor the most CTAs is right for every shape:
//   * the main loop is the slowest of: the multiplications of a rank's K blocks; all CTAs' bytes at what L2 delivers
//     (weights re-read by every pixel tile); the layer's weights, cold in HBM.  Where two are close they add up (a 4-norm);
//   * K blocks beyond the ring wait for their refill, and a deep ring of small tiles gains;
//   * the exchange of a K split costs its latency and the bytes that distributed shared memory takes, 15 a clock and SM; the
//     cluster barrier of a receive area over the ring;
//   * each turn of the two halves of a CTA over its pixel groups, more with a residual, a second output or GELU;
//   * a second CTA on an SM (it delays the early start of the next kernel), and every CTA a little.
// The constants were fitted on a B200, for the choice rather than the time: first to 6660 launches timed by themselves (316
// layers of ResNet, Inception, VGG, DenseNet and BERT at odd and even sizes, weights cold: on layers left out of the fit the choice
// is within 3 % of the best of a layer's ~20 plans, where the estimate for the staged exchange loses 7 %), then to 3655 replays of
// each of 21 whole models under different plans, where branches share the SMs and the next layer's weights load beside this
// one: 1.1 % faster over the models again (Inception-v3 5 %).
static float tc_plan_cycles(const ConvP& p, const TcPlan& c) {
    auto pow4 = [](float x) { return x * x * x * x; };
    const float kb = (float)c.kb_per_split, rows = (float)(p.co < TC_BM ? ceil_div_i(p.co, 8) * 8 : TC_BM);
    const float bytes = 128.f * (rows + c.n_valid), ctas = (float)c.splits * c.n_tiles * c.m_tiles;
    const float weights = 4.f * p.co * p.ci * p.kh * p.kw;
    const float mma = 189.f + 0.273f * c.n_mma;
    float t = sqrtf(sqrtf(pow4(kb * (mma > 2.f * c.n_mma ? mma : 2.f * c.n_mma)) + pow4(ctas * kb * bytes / 22500.f) + pow4(weights / 4460.f)));
    t += (411.f * (c.kb_per_split - c.stages) + 67.f * kb) / c.stages;
    if (c.splits > 1)
        t += 1210.f + 51.f * c.recv_late + 0.317f * c.n_valid * (p.co < TC_BM ? p.co : TC_BM) * (c.splits - 1) / c.splits;
    const int groups = ceil_div_i(c.n_valid, 4), turns = ceil_div_i(c.gpc < groups ? c.gpc : groups, 2);
    t += turns * (606.f + (p.ep & EP_RES ? 203.f : 0.f) + (p.ep & EP_DUAL ? 106.f : 0.f) + (p.ep & EP_GELU ? 211.f : 0.f));
    return t + 0.79f * c.n_valid + 15.2f * ctas + 1760.f * (ceil_div_i((int)ctas, 148) - 1);
}

// The estimate that chose plans when partials were read from the peers' staging tiles.  Schedules written then state its choice and
// load with it (see ConvP::plan_earlier).
static float tc_plan_cycles_earlier(const ConvP& p, const TcPlan& c) {
    auto pow4 = [](float x) { return x * x * x * x; };
    const float kb = (float)c.kb_per_split, bytes = TC_A_BYTES + 128.f * c.n_valid;
    const float ctas = (float)c.splits * c.n_tiles * c.m_tiles;
    const float weights = 4.f * p.co * p.ci * p.kh * p.kw;
    const float row_turns = (float)ceil_div_i(c.cpc_max, 8);   // turns of eight warps, a pixel row each
    float t = sqrtf(sqrtf(pow4(kb * 75.f) + pow4(ctas * kb * bytes / 7000.f) + pow4(weights / 720.f)));
    t += 760.f * kb / c.stages + 25.f * c.n_valid + ctas;
    if (c.splits > 1) t += 450.f + 38.f * c.splits;
    if (p.ep & EP_RES) t += 300.f * row_turns;
    if (p.ep & EP_GELU) t += 300.f * row_turns;
    return t + 1570.f * (ceil_div_i((int)ctas, 148) - 1);
}

// The plan of a layer: of the tile caps and K splits that fit, the one with the least estimated time.  A kernel name can fix
// a measured plan instead (tp = tile cap, ts = K splits, written by the resource generator; reef_b200/tune.py).
int tc_plan(const ConvP& p, TcPlan* pl) {
    if (p.nchw || (p.ci & 3) || p.ci < 4 || p.sh != p.sw || (p.sh != 1 && p.sh != 2)) return REEF_NOT_FOUND;
    if ((p.ics & 3) || (p.ioff & 3) || (p.ocs & 3) || (p.ooff & 3) || (p.co & 3)) return REEF_NOT_FOUND;
    if (p.kh * p.kw > 64) return REEF_NOT_FOUND;
    if (p.plan_cap > 0) {
        // tile cap fixed by the kernel name (a tuned plan): that candidate or nothing
        if (p.plan_cap < 8 || p.plan_cap > 208) return REEF_NOT_FOUND;
        const int rc = tc_plan_cap(p, p.plan_cap, p.plan_splits, pl);
        return rc == REEF_SUCC ? tc_place_recv(pl, p.plan_earlier != 0) : rc;
    }
    TcPlan best;
    float best_cycles = 0.f;
    const bool earlier = p.plan_earlier != 0;
    for (int cap : {208, 160, 128, 112, 96, 80, 64, 56, 48, 40, 32, 24, 16, 8}) {
        if (earlier && (cap == 56 || cap == 40 || cap == 8)) continue;
        for (int want = 1; want <= TC_MAX_SPLITS; want *= 2) {
            const int fixed = p.plan_splits;   // a name may fix the splits alone: as many of them as K allows
            if (fixed > 0 && want > 1) break;
            TcPlan c;
            if (tc_plan_cap(p, cap, fixed > 0 ? fixed : want, &c) != REEF_SUCC) continue;
            if (fixed == 0 && c.splits != want) continue;
            float cycles = earlier ? tc_plan_cycles_earlier(p, c) : 0.f;   // (its ring was not yet shared with a receive area)
            if (tc_place_recv(&c, earlier) != REEF_SUCC) continue;
            if (!earlier) cycles = tc_plan_cycles(p, c);
            if (best_cycles == 0.f || cycles < best_cycles) {
                best = c;
                best_cycles = cycles;
            }
        }
    }
    if (best_cycles == 0.f) return REEF_NOT_FOUND;
    *pl = best;
    return REEF_SUCC;
}

// ---- tensor maps ---------------------------------------------------------------------------------
typedef CUresult (*encode_tiled_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static encode_tiled_fn g_encode = nullptr;

static int get_encode() {
    if (g_encode) return REEF_SUCC;
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn) {
        set_error("cuTensorMapEncodeTiled is not available from the driver");
        return REEF_FAIL;
    }
    g_encode = (encode_tiled_fn)fn;
    return REEF_SUCC;
}

static int encode(CUtensorMap* tm, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides_bytes,
                  const cuuint32_t* box) {
    cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    CUresult r = g_encode(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (cuuint32_t)rank, const_cast<void*>(base), dims,
                          strides_bytes, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed with CUresult " + std::to_string((int)r));
        return REEF_FAIL;
    }
    return REEF_SUCC;
}

// The error word is pinned host memory mapped into the device's address space: a kernel whose bounded wait
// expired stores 1 through the device pointer, the host reads the word directly once the stream is synchronised.
static int* g_error_word[16] = {nullptr};        // device view
static int* g_error_word_host[16] = {nullptr};   // host view of the same word

int tc_error_word(int** out) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 16) return REEF_FAIL;
    if (!g_error_word[dev]) {
        int* h = nullptr;
        int* d = nullptr;
        if (cudaHostAlloc((void**)&h, 64, cudaHostAllocMapped) != cudaSuccess ||
            cudaHostGetDevicePointer((void**)&d, h, 0) != cudaSuccess) {
            set_error("cannot allocate the device error word");
            return REEF_FAIL;
        }
        *h = 0;
        g_error_word_host[dev] = h;
        g_error_word[dev] = d;
    }
    *out = g_error_word[dev];
    return REEF_SUCC;
}

int tc_error_word_host(volatile int** out) {
    int* d = nullptr;
    int rc = tc_error_word(&d);
    if (rc != REEF_SUCC) return rc;
    int dev = 0;
    cudaGetDevice(&dev);
    *out = g_error_word_host[dev];
    return REEF_SUCC;
}

int tc_build_params(const ConvP& p, const TcPlan& pl, void* const* a, TcParams* P) {
    int rc = get_encode();
    if (rc != REEF_SUCC) return rc;
    memset(P, 0, sizeof(*P));
    const float* in = (const float*)a[0];
    const float* wgt = (const float*)a[1];
    {
        // weights [Cout][tap][Cin] as a 3-d map (Cin, taps, Cout): a box is 32 channels of one tap for 128 output
        // channels, and channels beyond Cin (Cin not a multiple of 32) come back as zeros
        cuuint64_t dims[3] = {(cuuint64_t)p.ci, (cuuint64_t)(p.kh * p.kw), (cuuint64_t)p.co};
        cuuint64_t strides[2] = {(cuuint64_t)p.ci * 4, (cuuint64_t)p.ktot * 4};
        // Fewer output channels than a tile has rows: only they are copied (in whole 8-row groups of the swizzle).  The
        // other rows of the operand keep what the shared memory held; their sums end in lanes that nobody reads.
        const cuuint32_t rows = p.co < TC_BM ? (cuuint32_t)ceil_div_i(p.co, 8) * 8 : TC_BM;
        P->load_bytes = (int)rows * TC_BK * 4 + pl.b_bytes;
        cuuint32_t box[3] = {TC_BK, 1, rows};
        rc = encode(&P->tm_w, wgt, 3, dims, strides, box);
        if (rc != REEF_SUCC) return rc;
    }
    if (pl.spatial) {
        const int s = p.sh;
        for (int ry = 0; ry < s; ry++)
            for (int rx = 0; rx < s; rx++) {
                const int nx = (p.wi - rx + s - 1) / s, ny = (p.hi - ry + s - 1) / s;
                if (nx <= 0 || ny <= 0) continue;
                const float* base = in + p.ioff + ((size_t)ry * p.wi + rx) * p.ics;
                cuuint64_t dims[3] = {(cuuint64_t)p.ci, (cuuint64_t)nx, (cuuint64_t)ny};
                cuuint64_t strides[2] = {(cuuint64_t)s * p.ics * 4, (cuuint64_t)s * p.wi * p.ics * 4};
                cuuint32_t box[3] = {TC_BK, (cuuint32_t)pl.xw, (cuuint32_t)pl.rows};
                rc = encode(&P->tm_x[ry * s + rx], base, 3, dims, strides, box);
                if (rc != REEF_SUCC) return rc;
            }
    } else {
        cuuint64_t dims[2] = {(cuuint64_t)p.ci, (cuuint64_t)p.ptot};
        cuuint64_t strides[1] = {(cuuint64_t)p.ics * 4};
        cuuint32_t box[2] = {TC_BK, (cuuint32_t)pl.n_valid};
        rc = encode(&P->tm_x[0], in + p.ioff, 2, dims, strides, box);
        if (rc != REEF_SUCC) return rc;
    }
    P->out = (float*)a[2];
    P->res = (p.ep & EP_RES) ? (const float*)a[p.i_res] : nullptr;
    P->bias = (p.ep & EP_BIAS) ? (const float*)a[p.i_bias] : nullptr;
    P->gamma = (p.ep & EP_GB) ? (const float*)a[p.i_gamma] : nullptr;
    P->beta = (p.ep & EP_GB) ? (const float*)a[p.i_beta] : nullptr;
    P->out2 = (p.ep & EP_DUAL) ? (float*)a[p.i_out2] : nullptr;
    P->bias2 = (p.ep & EP_DUAL) ? (const float*)a[p.i_bias2] : nullptr;
    P->pcs = p.pcs; P->poff = p.poff;
    rc = tc_error_word(&P->error_word);
    if (rc != REEF_SUCC) return rc;
    P->co = p.co; P->ci = p.ci; P->ptot = p.ptot; P->ocs = p.ocs; P->ooff = p.ooff;
    P->spatial = pl.spatial; P->wo = p.wo; P->rows = pl.rows; P->xsplit = pl.xsplit; P->xw = pl.xw;
    P->n_valid = pl.n_valid; P->n_mma = pl.n_mma; P->tmem_cols = pl.tmem_cols;
    P->kh = p.kh; P->kw = p.kw; P->stride = p.sh; P->ph = p.ph; P->pw = p.pw;
    P->cblocks = pl.cblocks; P->kb_total = pl.kb_total; P->kb_per_split = pl.kb_per_split; P->splits = pl.splits;
    P->ep = 0;
    if (p.ep & EP_RES) P->ep |= TC_EP_RES;
    if (p.ep & EP_BIAS) P->ep |= TC_EP_BIAS;
    if (p.ep & EP_GB) P->ep |= TC_EP_GB;
    if (p.ep & EP_RELU) P->ep |= TC_EP_RELU;
    if (p.ep & EP_GELU) P->ep |= TC_EP_GELU;
    if (p.round_tf32) P->ep |= TC_EP_ROUND;
    P->cb_magic = (unsigned)((0x100000000ull + (unsigned long long)pl.cblocks - 1) / (unsigned long long)pl.cblocks);
    for (int ky = 0; ky < p.kh; ky++)
        for (int kx = 0; kx < p.kw; kx++) {
            const int s = p.sh, dy = ky - p.ph, dx = kx - p.pw;
            const int ry = ((dy % s) + s) % s, rx = ((dx % s) + s) % s;
            const int tap = ky * p.kw + kx;
            P->tap_map[tap] = (signed char)(ry * s + rx);
            P->tap_qx[tap] = (signed char)((dx - rx) / s);
            P->tap_qy[tap] = (signed char)((dy - ry) / s);
        }
    P->stages = pl.stages;
    P->region_bytes = pl.region_bytes;
    P->recv_offset_floats = pl.recv_offset_floats;
    P->cpc_max = pl.cpc_max;
    P->gpc = pl.gpc;
    P->gpc_magic = (unsigned)((65536 + pl.gpc - 1) / pl.gpc);
    P->recv_offset = pl.recv_offset;
    P->recv_late = pl.recv_late;
    P->n_tiles = pl.n_tiles;
    P->tile_begin = 0;
    P->pdl = 1;
#ifdef REEF_DEBUG_AIDS
    P->withheld_rank = P->withheld_load = -1;   // (no delay either)
#endif
    return REEF_SUCC;
}

static bool g_attr_set[16] = {false};

// The number of K splits is a template parameter: the exchange and the sums are straight code behind the accumulator.
typedef void (*tc_kernel_fn)(TcParams);
static tc_kernel_fn tc_kernel(bool be, int splits) {
    switch (splits) {
        case 1: return be ? reef_conv_tc_kernel<true, 1> : reef_conv_tc_kernel<false, 1>;
        case 2: return be ? reef_conv_tc_kernel<true, 2> : reef_conv_tc_kernel<false, 2>;
        case 4: return be ? reef_conv_tc_kernel<true, 4> : reef_conv_tc_kernel<false, 4>;
        default: return be ? reef_conv_tc_kernel<true, 8> : reef_conv_tc_kernel<false, 8>;
    }
}

#ifdef REEF_DEBUG_AIDS
static long long* g_trace[16] = {nullptr};
// Phase trace of the tensor-core convolution (development builds only): when enabled, block (0,0) of every launch
// stamps the SM clock at 11 points (entry, set-up done, ring filled, peers up, first K block landed, last K block
// landed, accumulator complete, tile staged, exchange complete, rows finished, TMEM freed) into one 16-word device
// record that the host reads back.
int tc_trace_enable(int on) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 16) return REEF_FAIL;
    if (on && !g_trace[dev]) {
        if (cudaMalloc(&g_trace[dev], 128) != cudaSuccess || cudaMemset(g_trace[dev], 0, 128) != cudaSuccess) {
            set_error("cannot allocate the trace record");
            return REEF_FAIL;
        }
    } else if (!on && g_trace[dev]) {
        cudaFree(g_trace[dev]);
        g_trace[dev] = nullptr;
    }
    return REEF_SUCC;
}
int tc_trace_read(long long* out16) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 16 || !g_trace[dev]) return REEF_NOT_FOUND;
    if (cudaMemcpy(out16, g_trace[dev], 128, cudaMemcpyDeviceToHost) != cudaSuccess) return REEF_FAIL;
    return REEF_SUCC;
}
#endif

// Programmatic dependent launch is on (development builds can switch it off with REEF_PDL=0, and for padded
// best-effort pieces alone with REEF_PAD_PDL=0).
static bool env_flag_on(const char* name) {
#ifdef REEF_DEBUG_AIDS
    const char* v = getenv(name);
    return !(v && v[0] == '0');
#else
    (void)name;
    return true;
#endif
}

// one-time, per device: shared-memory opt-in of both flavours of the kernel and the error word (never during a capture)
int tc_prepare_device() {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 16 && !g_attr_set[dev]) {
        for (int i = 0; i < 8; i++) {
            const void* fn = (const void*)tc_kernel(i & 1, 1 << (i >> 1));
            cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
            if (e == cudaSuccess)   // the whole unified L1/shared array as shared memory, so that two CTAs are resident
                e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
            if (e != cudaSuccess) {
                set_error(std::string("cudaFuncSetAttribute(conv_tc): ") + cudaGetErrorString(e));
                return REEF_FAIL;
            }
        }
        int* w = nullptr;
        int rc = tc_error_word(&w);
        if (rc != REEF_SUCC) return rc;
        g_attr_set[dev] = true;
    }
    return REEF_SUCC;
}

int tc_launch(const TcParams& P0, const TcPlan& pl, cudaStream_t st, const int* flag, int* slot, int tile_begin,
              int tile_count) {
    static const bool use_pdl = env_flag_on("REEF_PDL"), pad_pdl = env_flag_on("REEF_PAD_PDL");
    TcParams P = P0;
    P.preempt_flag = flag;
    P.task_slot = slot;
    const int tiles = pl.n_tiles * pl.m_tiles;
    if (tile_count < 0) tile_count = tiles - tile_begin;
    if (tile_begin < 0 || tile_count <= 0 || tile_begin + tile_count > tiles) {
        set_error("tensor-core convolution: tile range outside the kernel");
        return REEF_OUT_OF_RANGE;
    }
    P.tile_begin = tile_begin;
    P.stamps = flag != nullptr ? preempt_stamps_ptr() : nullptr;
    P.trace = nullptr;
#ifdef REEF_DEBUG_AIDS
    {
        int dev = 0;
        cudaGetDevice(&dev);
        P.trace = (dev >= 0 && dev < 16) ? g_trace[dev] : nullptr;
    }
#endif
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(pl.splits, tile_count, 1);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = st;
    cudaLaunchAttribute attrs[2];
    int na = 0;
    if (pl.splits > 1) {
        attrs[na].id = cudaLaunchAttributeClusterDimension;
        attrs[na].val.clusterDim.x = pl.splits;
        attrs[na].val.clusterDim.y = 1;
        attrs[na].val.clusterDim.z = 1;
        na++;
    }
    const bool piece = flag == nullptr && slot != nullptr;   // a padded best-effort piece
    if (use_pdl && (!piece || pad_pdl)) {
        attrs[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attrs[na].val.programmaticStreamSerializationAllowed = 1;
        na++;
    }
    cfg.attrs = attrs;
    cfg.numAttrs = na;
    // the best-effort flavour (flag polls at block entry and at the producer's loop head) is its own instantiation:
    // the real-time flavour carries no poll
    cudaError_t e = cudaLaunchKernelEx(&cfg, tc_kernel(flag != nullptr, pl.splits), P);
    if (e != cudaSuccess) {
        set_error(std::string("cudaLaunchKernelEx(conv_tc): ") + cudaGetErrorString(e));
        return REEF_FAIL;
    }
    return REEF_SUCC;
}

int tc_func_attrs(const TcPlan& pl, cudaFuncAttributes* fa, int* occ) {
    cudaError_t e = cudaFuncGetAttributes(fa, (const void*)tc_kernel(false, pl.splits));
    if (e != cudaSuccess) {
        set_error(std::string("cudaFuncGetAttributes(conv_tc): ") + cudaGetErrorString(e));
        return REEF_FAIL;
    }
    // shared memory (plus the 1 KB the hardware reserves per CTA) and 128 registers x 256 threads: two at most
    const int by_smem = (228 * 1024) / (pl.smem + 1024);
    *occ = by_smem < 1 ? 1 : (by_smem > 2 ? 2 : by_smem);
    return REEF_SUCC;
}

}  // namespace reef
