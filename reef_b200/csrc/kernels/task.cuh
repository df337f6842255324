// Shared device-side vocabulary of the kernel registry.
//
// Every kernel family is written once as a __device__ body that executes ONE logical thread
// block ("vblock") of 256 threads.  Three __global__ flavours wrap the same body, mirroring the
// three code objects the reference builds per model (reference: resource/Makefile:22-66):
//   plain      one CUDA block per vblock                       (<m>.raw.co)
//   best-effort  plain + preempt-flag poll + completion counter (<m>.be.co,
//              reference: script/best_effort_kernel.py:22-33)
//   dispatcher a persistent grid that pulls vblocks of a real-time and a best-effort
//              kernel (<m>.trans.co, reference: resource/mocked_kernel/mocked_kernel.trans.cu:112-186)
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace reef {

constexpr int kThreads = 256;   // every family runs 256-thread blocks so the dispatcher can host any of them
constexpr int kMaxArgs = 8;

enum Family : int {
    F_MOCK_ADD = 0,
    F_MOCK_MUL,
    F_FUSED_ADD_NCHW,
    F_BIAS_RELU,
    F_CONV_SIMT,
    F_MAX_POOL,
    F_AVG_POOL,
    F_GLOBAL_AVG_POOL,
    F_COPY,
    F_DENSE,
    F_SOFTMAX,
    F_EMBEDDING,
    F_LAYERNORM,
    F_ATTENTION,
    F_ATTENTION_STAGED,
    F_NCHW_TO_NHWC4,
    F_IM2COL_NCHW,
    F_COUNT,
    // families with their own __global__ kernel (not hosted by the 256-thread logical-block wrappers)
    F_CONV_TC = 100,
    F_ATTENTION_TC = 101
};

// epilogue / option bits
enum : int { EP_RES = 1, EP_BIAS = 2, EP_GB = 4, EP_RELU = 8, EP_GELU = 16, EP_DUAL = 32 };

struct ConvP {
    int ci, hi, wi, co, kh, kw, sh, sw, ph, pw, ho, wo;
    int ics, ioff, ocs, ooff, nchw;
    int ktot, ptot;          // K = kh*kw*ci, P = ho*wo
    int tiles_p, tiles_c;    // tile grid: pixels x out-channels
    int tile_c, kgroups;     // fp32 variant: channels of a warp tile (32 or 16), warps sharing a tile's K
    int ep;                  // EP_* bits
    int i_res, i_bias, i_gamma, i_beta;   // positions in the arg list, -1 when absent
    int round_tf32;          // tensor-core variant: store activations rounded to the nearest TF32 value
    int i_bias2, i_out2;     // EP_DUAL: second output out2 = relu(out + bias2) (the next unit's pre-activation)
    int pcs, poff;           // channel stride and offset of the second output
    int plan_cap, plan_splits;   // tensor-core variant: tile cap / K splits fixed by the name (tp, ts), 0 = planner's choice
    int plan_earlier;            // tensor-core variant: the plan that earlier versions wrote into schedules (pv1)
};

struct PoolP {
    int c, hi, wi, k, s, p, ho, wo, ics, ioff, ocs, ooff, cip, has_bias;
};

struct EltP {
    int c, n, ics, ioff;     // channels, rows (pixels) ; NCHW fused_add: c planes of n elements
    int ocs, ooff;           // fused_add_nn_relu: channel stride and offset of the output
};

struct DenseP {
    int k, n, relu;
};

struct SoftmaxP {
    int rows, n;
};

struct KTask {
    int family;
    int nblocks;             // logical blocks of one launch
    union {
        ConvP conv;
        PoolP pool;
        EltP elt;
        DenseP dense;
        SoftmaxP softmax;
        int raw[32];
    } p;
    void* a[kMaxArgs];       // device pointers, positional like the json "args"
    int* err;                // device error word (set when a bounded wait expired), may be null
};

__device__ __forceinline__ int ld_flag(const int* flag) {
    return *reinterpret_cast<const volatile int*>(flag);
}

// Programmatic dependent launch: this kernel waits for its predecessor's results before touching memory (a
// no-op for an ordinary launch) and only then lets its successor start its prologue.  Releasing the successor
// before the wait would let a chain of kernels run ahead without bound: every grid's blocks would become
// resident, release the next grid and park at their wait, until the SMs are full of parked blocks and a
// best-effort kernel on another stream finds no room.  In this order at most two grids of a chain are resident.
__device__ __forceinline__ void pdl_prologue() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// How a block enters: called once, with all threads, ahead of a body's first access to memory.  The fp32 convolution calls it
// itself, behind what it works out from its parameters: its divisions and addresses, half a microsecond of a launch, are then out
// of the way while the previous kernel still runs (5 % of a replay of ResNet-50 at 193x193, 8 % at 70x70).  The other bodies have
// little to work out: it is called ahead of them (inside pooling, elementwise kernels, the im2col gather, LayerNorm and attention no
// model gained).  False: leave.
struct EnterAlways {        // the dispatcher's blocks
    __device__ __forceinline__ bool operator()() const { return true; }
};
struct EnterPlain {
    __device__ __forceinline__ bool operator()() const {
        pdl_prologue();
        return true;
    }
};
// Best-effort: ONE thread reads the flag and the block takes one decision: were every thread to read it for itself, a flag
// that goes up between the reads of two warps would let part of a block leave and the rest run the body with
// threads missing (wrong partial sums counted as a complete block, barriers short of arrivals).  It is read ahead of
// the wait for the previous kernel, so that its trip to L2 (0.4 us) is not on the way to the body: a flag that goes up
// during that wait is seen by the body's polls or by the next kernel of the stream, which starts behind this wait.  A body without
// polls then runs whole behind a kernel that left early, over partial data, and counts its block: the run is
// resumed from the first short counter, and what later counters say means nothing.
struct EnterBestEffort {
    int up;                 // what thread 0 read, 0 elsewhere
    __device__ __forceinline__ bool operator()() const {
        pdl_prologue();
        return !__syncthreads_or(up);
    }
};

}  // namespace reef
