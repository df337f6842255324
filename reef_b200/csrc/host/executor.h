// Executors: own a model's device storage and launch its kernels through the C-ABI device layer.
//
//   ExecutorBase   raw kernels in json order                 (reference: src/reef/executor/executor_base.{h,cpp})
//   HybridExecutor + per-kernel scheduling metadata (KernelArg: logical blocks, minimal occupancy,
//                  resources, latency profile), the best-effort flavour with preempt flag and
//                  completion counters, the dispatcher launch, and a CUDA-graph fast path
//                  (reference: src/reef/executor/trans_executor.{h,cpp}, hybrid_executor.{h,cpp})
#pragma once
#include <atomic>
#include <memory>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../../include/reef_cuda.h"
#include "common.h"
#include "model.h"

namespace reef {
namespace server {
class REEFScheduler;
}
namespace executor {

typedef reef_dptr_t GPUDevicePtr_t;
typedef reef_kernel_t GPUFunction_t;
typedef reef_module_t GPUModule_t;
typedef reef_stream_t GPUStream_t;

class ExecutorBase {
public:
    ExecutorBase();
    virtual ~ExecutorBase();

    // co_file_path is accepted for signature parity; kernels come from the built-in registry.
    Status load_model_from_file(const char* json_file_path, const char* co_file_path = nullptr);
    virtual Status load_model_from_GPU_module(const char* json_file_path, GPUModule_t module);
    Status load_param_from_file(const char* param_file_path);

    Status set_input(const std::string& key, const std::vector<float>& value);
    Status set_input(int idx, const void* value, size_t len);
    Status set_input(const std::string& key, const void* value, size_t len);
    Status get_data_size(const std::string& key, size_t& size);
    Status get_output(std::vector<float>& out);
    Status get_output(void* out, size_t len);
    Status get_data(int idx, void* out, size_t len);
    // asynchronous I/O on a stream from/to pinned host memory (no reference counterpart: the
    // reference copies synchronously on the default stream, executor_base.cpp:112-116)
    Status set_input_async(const std::string& key, const void* value, size_t len, GPUStream_t stream);
    Status get_output_async(void* out, size_t len, GPUStream_t stream);

    Status execute(GPUStream_t stream = nullptr);
    Status execute_to(int idx, GPUStream_t stream = nullptr);
    Status execute_kernel(int idx, GPUStream_t stream = nullptr);
    Status execute_kernel_async(int idx) {   // no sync
        drop_output_mirror();
        return launch_kernel(idx, s);
    }
    size_t num_kernels() const;
    // name of kernel i as the schedule gives it (diagnostics)
    const char* kernel_name(size_t i) const { return model && i < model->kernels.size() ? model->kernels[i].name.c_str() : "?"; }

    void set_stream(GPUStream_t stream);
    GPUStream_t stream() const;
    const std::string& error() const { return err_; }
    // Failure injection on the host: the next `n` kernel launches of this executor return Status::Fail without
    // reaching the device (how the tests exercise the failed-task path; no GPU fault is involved).
    void inject_launch_failures(int n) { fail_launches = n; }
    // the same for the next `n` launches of the output mirror (launch_output_mirror)
    void inject_mirror_failures(int n) { fail_mirrors = n; }

    // The output tensor of a complete run, already in host memory: every full pass ends with a copy of "output" into a
    // pinned mirror on the pass's own stream, so that get_output behind the pass is a plain memcpy.  `launch` enqueues
    // that copy; `drop` says that the device tensor may have changed since (get_output then copies it itself).
    Status launch_output_mirror(GPUStream_t stream);
    void drop_output_mirror() { mirror_fresh.store(false, std::memory_order_relaxed); }
    // makes `stream` wait for a set_input whose copy may still be under way (no host wait); called by everything that
    // launches kernels of this executor
    Status order_input(GPUStream_t stream);

    std::unique_ptr<Model> model;
    static Status resolve_kernels(const Model& m, GPUModule_t mod, std::vector<GPUFunction_t>* out_kernels,
                                  std::vector<uint32_t>* out_smem, std::string* err);

protected:
    Status init_executor_base(const char* json_file_path, GPUModule_t module);
    virtual Status launch_kernel(int kernel_offset, GPUStream_t stream);
    Status find_storage_idx(const std::string& name, size_t& idx);
    size_t storage_bytes(size_t idx) const;
    Status init_host_buffers();
    Status wait_input();
    // the bare launches, as a capture records them: no order behind an input, no failure injection, no note of the mirror
    Status issue_kernel(int kernel_offset, GPUStream_t stream);
    Status issue_mirror(GPUStream_t stream);

    std::vector<GPUDevicePtr_t> storage;            // one device pointer per storage entry (views into one arena)
    std::vector<GPUFunction_t> kernels;             // per kernel call
    std::vector<uint32_t> kernel_smem;              // per kernel call, from "shared_memory"
    std::vector<std::vector<void*>> raw_args;       // raw_args[k][j] = &storage[idx]
    GPUDevicePtr_t arena = 0;
    size_t arena_bytes = 0;
    GPUModule_t base_mod = nullptr;
    bool own_module = false;
    GPUStream_t s = nullptr;
    std::unordered_map<std::string, size_t> storage_idx;   // name -> first storage entry of that name
    // host side of a request: one pinned allocation = input staging area | output mirror
    unsigned char* host_buf = nullptr;
    size_t stage_bytes = 0;
    unsigned char* mirror = nullptr;
    reef_event_t input_ev = nullptr;                // behind the last staged input copy
    std::atomic<bool> input_pending{false};         // some stream has yet to be ordered behind input_ev
    GPUStream_t input_stream = nullptr;
    size_t mirror_bytes = 0;
    reef_kernel_t mirror_kernel = nullptr;          // device -> mapped host copy of "output" (null: the copy engine's)
    uint32_t mirror_dims[6] = {0, 0, 0, 0, 0, 0};
    uint32_t mirror_smem = 0;
    GPUDevicePtr_t mirror_args[2] = {0, 0};
    std::atomic<bool> mirror_fresh{false};
    int fail_launches = 0;
    int fail_mirrors = 0;
    std::string err_;
};

class HybridExecutor : public ExecutorBase {
    friend class server::REEFScheduler;

public:
    // reference: trans_executor.h:47-63
    class KernelArg {
    public:
        int block_num = 0;        // logical thread blocks of the kernel
        int block_offset = 0;
        int threads = 0;
        int min_occupancy = 1;    // minimal blocks/SM the real-time kernel needs to finish in one wave
        int granularity = 1;      // block ranges handed to the dispatcher are multiples of this (cluster size)
        reef_kernel_attrs_t resource{};
        KernelProfile profile;
    };

    HybridExecutor();
    virtual ~HybridExecutor();

    // The three code-object paths of the reference signature are accepted and ignored.
    Status load_hybrid_model_from_file(const char* json_file_path, const char* profile_file_path,
                                       const char* trans_co_file_path = nullptr,
                                       const char* preempt_co_file_path = nullptr);

    Status execute_preemptale(GPUStream_t stream = nullptr);     // (sic) reference spelling
    Status set_preempt_flag(GPUDevicePtr_t flag);
    Status reset_task_slot_async(int kernel_offset, GPUStream_t stream);
    void reset_task_slots(GPUStream_t stream, int from_kernel = 0);
    void copy_be_kernel_offset(GPUStream_t stream);
    // Where a preempted run restarts: the first kernel from `begin` on whose counter is short of its block count.  What the
    // counters behind it say means nothing: a block decides whether to run from a look at the flag that was taken ahead of its
    // wait for the kernel before, so a kernel behind one that left early may run whole, over partial data, and count every block.
    int get_be_kernel_offset(int begin);
    const std::vector<int>& preempted_slots() const { return preempted_slots_; }

    Status launch_preempt_kernel(int kernel_offset, GPUStream_t stream);
    // dispatcher launch of kernel `rt_idx`, padded with logical blocks of `be`'s kernel `be_idx`
    // `be_stream` non-null (or a tensor-core kernel on either side): the best-effort blocks are launched
    // beside the real-time kernel on be_stream instead of inside one grid
    Status launch_dispatch(int rt_idx, HybridExecutor* be, int be_idx, int be_block_offset, int be_block_num,
                           int sm_partition, int occupancy, GPUStream_t stream, GPUStream_t be_stream = nullptr);
    // best-effort logical blocks [offset, offset+num) of kernel idx alone, non-preemptible, counted into the task slot
    Status launch_pad_piece(int idx, int block_offset, int block_num, int occupancy, GPUStream_t stream);
    // Padding segments: the kernel list cut into runs of kPadSegment kernels, each run captured once as a CUDA
    // graph of whole-kernel pieces (one launch and one completion event for the run; inside it the kernels keep
    // their programmatic dependencies).  Segment g covers kernels [g*kPadSegment, (g+1)*kPadSegment).
    // They are captured on `cap`, a stream with nothing on it: a graph's kernels keep the priority and the SM partition of
    // the stream that they were captured on, wherever the graph is launched.
    static const int kPadSegment = 4;
    Status build_pad_segments(GPUStream_t cap);
    bool has_pad_segments() const { return !pad_segments.empty(); }
    Status launch_pad_segment(int seg, GPUStream_t stream);
    // Best-effort segments: the same cut into runs of kBeSegment kernels for the best-effort flavour (every kernel still
    // polls the flag and counts into its slot).  A task at full speed is fed one graph launch and one event per run.
    // Padding and preemption leave a task at any multiple of kPadSegment: short runs take it to the next boundary of kBeSegment.
    // Kernel by kernel, they waited for a host that feeds all clients at 4 us a kernel, until the next real-time request was due
    // and no longer run at all: ResNet-50 at 224 px over four best-effort ResNet-18, all served, 904 -> 790 us, BERT-base with 77
    // tokens over four ResNet-50 1300 -> 1210.  Real-time latencies behind pauses of 0.3 to 5 ms are what they were.
    static const int kBeSegment = 16;
    static_assert(kBeSegment % kPadSegment == 0, "a short segment ends where a long one begins");
    Status build_be_segments(GPUStream_t cap);
    void drop_be_segments();
    Status launch_preempt_segment(int kernel_offset, GPUStream_t stream, bool single, int* last);
    bool has_tensor_core_kernels() const { return has_tc; }
    // Persistent chains: every run of two or more consecutive tensor-core convolution / matmul kernels of the
    // schedule becomes ONE persistent kernel (reef_chain_create) with `clusters` 8-CTA clusters (0 = the library's
    // default).  Built here, once; execute_graph and execute_chained then launch a run through its chain.  Results
    // are bit-identical to the per-kernel launches.  Call before the first execute_graph on a stream.
    Status build_chains(int clusters = 0);
    size_t num_chains() const { return chains.size(); }
    Status chain_info(size_t idx, int* begin, int* end, int* clusters, int* max_clusters) const {
        if (idx >= chains.size()) return Status::OutOfRange;
        int layers = 0;
        if (begin) *begin = chains[idx].begin;
        if (end) *end = chains[idx].end;
        GPU_RETURN_STATUS(reef_chain_info(chains[idx].handle, &layers, clusters, max_clusters));
        return Status::Succ;
    }
    // the whole schedule with chains where they exist and plain launches elsewhere, then sync
    Status execute_chained(GPUStream_t stream = nullptr);
    // Best-effort flavour with chains: kernel `k` must be the first kernel of a chain or inside one; the chain is
    // launched from that layer on `clusters` clusters (0 = default) with the preempt flag polled at every tile.
    // Returns the chain's end (first kernel behind it) in *next.
    Status launch_preempt_chain(int k, int clusters, GPUStream_t stream, int* next);
    // chain index whose run contains kernel k, or -1
    int chain_of(int k) const {
        for (size_t i = 0; i < chains.size(); i++)
            if (k >= chains[i].begin && k < chains[i].end) return (int)i;
        return -1;
    }
    // after a preemption: copy every chain's counters on `stream` (async); once the stream is synchronised,
    // chain_kernel_offset(from) = the first kernel at or behind `from` that is not known complete
    void copy_chain_progress(GPUStream_t stream);
    int chain_kernel_offset(int from);
    // best-effort flavour of the whole schedule, chains on `clusters` clusters, then sync (the flag is not touched)
    Status execute_preemptable_chained(int clusters, GPUStream_t stream = nullptr);
    // best-effort run of the whole schedule with chains, flag raised after delay_us, resumed until done
    Status execute_preempt_resume_chained(int delay_us, int clusters, int* restarts, int* first_incomplete);
    // execute_graph, then sync: repeated passes over a schedule do not pay for its launches one by one (an encoder of 16
    // small kernels: 77 us kernel by kernel, 67 us)
    Status execute(GPUStream_t stream = nullptr);
    // the whole kernel list on `stream`: launched kernel by kernel the first time, then captured as a CUDA graph and
    // replayed.  build_graph captures it ahead of the first pass, for launches on `stream`, on a stream `cap` of the same
    // kind with nothing on it: a server's requests then never wait for a capture.
    Status execute_graph(GPUStream_t stream);
    Status build_graph(GPUStream_t cap, GPUStream_t stream);
    bool has_graph(GPUStream_t stream) const { return graph != nullptr && graph_stream == stream; }
    // every kernel through the dispatcher without a best-effort partner, then sync
    Status execute_dispatch(GPUStream_t stream = nullptr);
    // best-effort run, flag raised delay_us after the first launch, resumed from the first incomplete kernel until done
    // (*first_count: the completion counter of that kernel when it was found short — between 0 and its block count)
    Status execute_preempt_resume(int delay_us, int* restarts, int* first_incomplete, int* first_count = nullptr);
    // device time of each kernel (us, CUDA events, average of iters)
    Status profile_kernels(int iters, float* us);
    // one persistent wave of kernel idx: sms*occupancy logical blocks through the dispatcher (us)
    Status profile_wave(int idx, int occupancy, int iters, float* us);
    // Measures the latency tables the padding policy reads (the reference's profile.json, produced there by a
    // `profiler` binary that is not in its tree, resource/Makefile:32-36): per distinct kernel name the average
    // duration of back-to-back launches (total_latency) and of one persistent wave at occupancy j+1
    // (latency[j]); model_latency = one graph replay.  All in nanoseconds (latency_unit_ns = 1).
    Status measure_profile(int iters, ModelProfile* out);
    const int* host_task_slots() const { return task_slots_host; }

    std::vector<KernelArg> trans_args;
    const ModelProfile* profile() const { return model_profile.get(); }

protected:
    Status init_hybrid_executor(const char* profile_file_path);

    GPUDevicePtr_t preempt_flag = 0;
    bool own_flag = false;
    GPUDevicePtr_t task_slot_base = 0;
    GPUDevicePtr_t dispatch_ctrl = 0;
    int* task_slots_host = nullptr;
    std::vector<int> preempted_slots_;   // counters found by the first preemption of execute_preempt_resume
    bool has_tc = false;
    std::shared_ptr<ModelProfile> model_profile;
    reef_graph_t graph = nullptr;
    std::vector<reef_graph_t> pad_segments;
    std::vector<reef_graph_t> be_segments;         // [k / kBeSegment]
    std::vector<reef_graph_t> be_short_segments;   // [k / kPadSegment], null at the boundaries of the long ones
    GPUStream_t graph_stream = nullptr;
    struct Chain {
        int begin, end;          // kernels [begin, end) of the schedule
        reef_chain_t handle;
    };
    std::vector<Chain> chains;
    Status launch_schedule(GPUStream_t stream, bool capturing);
    Status issue_preempt_kernel(int kernel_offset, GPUStream_t stream);
    Status issue_pad_piece(int idx, int block_offset, int block_num, int occupancy, GPUStream_t stream);
    // which launches of the schedule (and, as number num_kernels(), of the output mirror behind it) have to wait for
    // which others
    Status schedule_edges(std::vector<int>* from, std::vector<int>* to);
};

}  // namespace executor
}  // namespace reef
