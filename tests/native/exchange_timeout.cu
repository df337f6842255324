// The tensor-core convolution built with a short limit on its waits and with one load that is announced and never made
// (REEF_DEBUG_AIDS, REEF_WAIT_LIMIT_NS): what test_gpu_exchange_timeout.py runs.
#include "../../reef_b200/csrc/kernels/conv_tc.cu"

namespace reef {
void set_error(const std::string& s) { fprintf(stderr, "%s\n", s.c_str()); }
unsigned long long* preempt_stamps_ptr() { return nullptr; }
}  // namespace reef

// out[m][n] = x[m][k] * w[n][k]^T by tiles of `cap` pixels and `splits` ranks; rank `rank` of the first tile never gets its
// K block `load` (-1: it does) and, once it has given up, sends its shares `delay_ms` later.  plan[4] = {ranks, pixel tiles x channel tiles, K blocks of a rank, receive area over the ring}, slot = CTAs that counted themselves
// complete, error = the device error word, cleared again.
extern "C" __attribute__((visibility("default"))) int exchange_run(int m, int n, int k, int cap, int splits, int best_effort, int rank, int load, int delay_ms, const float* x,
                                                                   const float* w, float* out, int* plan, int* slot, int* error, float* ms) {
    using namespace reef;
    ConvP p;
    memset(&p, 0, sizeof(p));
    p.ci = k; p.hi = 1; p.wi = m; p.co = n; p.kh = p.kw = p.sh = p.sw = 1;
    p.ho = 1; p.wo = m; p.ics = k; p.ocs = n; p.pcs = n; p.ktot = k; p.ptot = m;
    p.plan_cap = cap; p.plan_splits = splits;
    TcPlan pl;
    if (tc_plan(p, &pl) != REEF_SUCC) return 1;
    plan[0] = pl.splits; plan[1] = pl.n_tiles * pl.m_tiles; plan[2] = pl.kb_per_split; plan[3] = pl.recv_late;
    float *dx, *dw, *dout;
    int* words;   // preempt flag, completion counter
    if (cudaMalloc(&dx, 4ull * m * k) || cudaMalloc(&dw, 4ull * n * k) || cudaMalloc(&dout, 4ull * m * n) || cudaMalloc(&words, 8)) return 2;
    if (cudaMemset(words, 0, 8) || cudaMemset(dout, 0, 4ull * m * n) || cudaMemcpy(dx, x, 4ull * m * k, cudaMemcpyHostToDevice) ||
        cudaMemcpy(dw, w, 4ull * n * k, cudaMemcpyHostToDevice))
        return 3;
    void* args[kMaxArgs] = {dx, dw, dout};
    TcParams P;
    if (tc_prepare_device() != REEF_SUCC || tc_build_params(p, pl, args, &P) != REEF_SUCC) return 4;
    P.withheld_rank = rank;
    P.withheld_load = load;
    P.withheld_delay_ns = delay_ms * 1000000;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    cudaEventRecord(a);
    const int rc = tc_launch(P, pl, nullptr, best_effort ? words : nullptr, words + 1);
    cudaEventRecord(b);
    if (rc != REEF_SUCC || cudaDeviceSynchronize() != cudaSuccess) return 5;
    cudaEventElapsedTime(ms, a, b);
    volatile int* word;
    if (tc_error_word_host(&word) != REEF_SUCC) return 6;
    *error = *word;
    *word = 0;
    if (cudaMemcpy(out, dout, 4ull * m * n, cudaMemcpyDeviceToHost) || cudaMemcpy(slot, words + 1, 4, cudaMemcpyDeviceToHost)) return 7;
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(dx); cudaFree(dw); cudaFree(dout); cudaFree(words);
    return 0;
}
