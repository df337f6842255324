"""Requests through host memory: staged input, output mirror, graph replay behind the first pass.  A one-kernel model that
copies its input makes every byte of the way visible; sizes straddle the two-piece split of the staging copy, the limit
between the mirror's copy kernel and the copy engine, and the limit of the pinned buffers."""
import ctypes as C
import threading

import numpy as np
import pytest

from reef_b200 import capi
from reef_b200.resources.graph import Graph, kname

pytestmark = pytest.mark.gpu

KB = 256            # floats per KB
SIZES = [1, 3, 128 * KB - 1, 128 * KB, 128 * KB + 5, 512 * KB, 512 * KB + 1, 4096 * KB, 4096 * KB + 3]


def copy_model(tmp_path, n):
    g = Graph("copy")
    data = g.input("data", n)
    g.kernel(kname("fused_nn_batch_flatten", n=n), [g.add_storage("output", n), data])
    return g.write(str(tmp_path), capi.plan_fn)


@pytest.mark.parametrize("n", SIZES)
def test_executor_request(tmp_path, n):
    base = copy_model(tmp_path, n)
    e = capi.HybridExecutor(0)
    e.load_model_from_file(base + ".json", base + ".profile.json")
    rng = np.random.default_rng(n)
    for run in (e.execute, e.execute_graph, e.execute_preemptable, e.execute_dispatch, lambda: e.execute_to(1)):
        for _ in range(3):      # plain launches, capture, replay
            x = rng.normal(0, 1, n).astype(np.float32)
            e.set_input("data", np.zeros(n, np.float32))
            e.set_input("data", x)      # the second input waits for the first one's copy
            run()
            assert np.array_equal(e.get_output(), x)
    e.set_input("data", x + 1)
    assert np.array_equal(e.get_output(), x), "a new input alone leaves the last output"
    assert np.array_equal(e.get_data(0, 4 * n), x + 1)
    e.close()


@pytest.mark.parametrize("kind", [capi.REEFScheduler.RealTimeQueue, capi.REEFScheduler.BestEffortQueue])
@pytest.mark.parametrize("n", [3, 128 * KB + 5, 512 * KB + 1, 4096 * KB + 3])
def test_scheduler_request(tmp_path, kind, n):
    base = copy_model(tmp_path, n)
    s = capi.REEFScheduler(capi.REEFScheduler.REEF, 0)
    mid = s.load_model_files(base + ".json", base + ".profile.json")
    s.bind_model_queue(s.create_queue(kind), mid)
    s.run()
    rng = np.random.default_rng(n)
    for _ in range(4):
        x = rng.normal(0, 1, n).astype(np.float32)
        s.set_input(mid, x)
        s.wait_task(s.new_task(mid))
        assert np.array_equal(s.get_output(mid), x)
    s.close()


@pytest.mark.parametrize("kernels", [1, 3, 4, 6])
def test_refused_output_mirror_of_a_padded_task(gen, tmp_path, kernels):
    """A best-effort task that goes out as padding beside a real-time request ends with the copy of its output into the
    pinned mirror.  Where that copy is refused the task is served all the same, and get_output must not hand out the
    answer of the request before (the copy is refused on the host; nothing fails on the device)."""
    n = 5000
    g = Graph("copies")
    src = g.input("data", n)
    for i in range(kernels):
        dst = g.add_storage("output" if i == kernels - 1 else "null", n)
        g.kernel(kname("fused_nn_batch_flatten", n=n), [dst, src])
        src = dst
    base, rt_base = g.write(str(tmp_path), capi.plan_fn), gen("resnet18_64")
    s = capi.REEFScheduler(capi.REEFScheduler.REEF, 0)
    s.set_pad_slowdown_target(0)      # no rate limit: whatever fits goes out as padding
    be = s.load_model_files(base + ".json", base + ".profile.json")
    rt = s.load_model_files(rt_base + ".json", rt_base + ".profile.json", rt_base + ".param")
    s.bind_model_queue(s.create_queue(capi.REEFScheduler.BestEffortQueue), be)
    s.bind_model_queue(s.create_queue(capi.REEFScheduler.RealTimeQueue), rt)
    s.set_input(rt, np.zeros(3 * 64 * 64, np.float32))
    s.run()
    rng = np.random.default_rng(kernels)
    refused = 0
    for i in range(40):
        x = rng.normal(0, 1, n).astype(np.float32)
        s.set_input(be, x)
        s.inject_mirror_failures(be, i % 2)
        # the second real-time request finds the best-effort task waiting and pads with it
        first, t, second = s.new_task(rt), s.new_task(be), s.new_task(rt)
        for task in (first, second):
            s.wait_task(task)
        try:
            s.wait_task(t)
        except capi.ReefError:      # not padded: the refused copy fails the task
            assert i % 2 and not s.get_task(t).padded_to_complete
            continue
        refused += i % 2 and s.get_task(t).padded_to_complete
        assert np.array_equal(s.get_output(be), x), f"request {i}: output of an earlier request"
    assert refused > 0
    s.close()


@pytest.mark.parametrize("kind", [capi.REEFScheduler.RealTimeQueue, capi.REEFScheduler.BestEffortQueue])
def test_input_set_while_graphs_are_captured(gen, kind):
    """A pipelined client stages inputs all the time.  One that arrives while a graph of the model is captured (by its first
    requests, or when it is bound) is no part of the capture: every request is served, and the input staged last counts."""
    base = gen("inception_v3_139")
    n = 3 * 139 * 139
    rng = np.random.default_rng(6)
    last = rng.normal(0, 1, n).astype(np.float32)
    want = None
    for _ in range(6):
        s = capi.REEFScheduler(capi.REEFScheduler.REEF, 0)
        mid = s.load_model_files(base + ".json", base + ".profile.json", base + ".param")
        q = s.create_queue(kind)
        s.run()
        stop, failed = threading.Event(), []

        def stage():
            x = rng.normal(0, 1, n).astype(np.float32)
            while not stop.is_set():
                try:
                    s.set_input(mid, x)
                except capi.ReefError as e:
                    failed.append(e)
                    return

        client = threading.Thread(target=stage)
        client.start()
        try:
            s.bind_model_queue(q, mid)
            for _ in range(6):
                s.wait_task(s.new_task(mid))
        finally:
            stop.set()
            client.join()
        assert not failed
        s.set_input(mid, last)
        s.wait_task(s.new_task(mid))
        out = s.get_output(mid)
        want = out if want is None else want
        assert np.array_equal(out, want)
        s.close()


@pytest.mark.parametrize("kernels", [1, 7, 8, 9, 16, 17])
def test_best_effort_segments(tmp_path, kernels):
    """Schedules shorter than, equal to and just beyond a segment of the best-effort window, with the GPU to themselves
    (whole segments) and while a real-time client is active (single kernels, resumed anywhere in a segment)."""
    n = 5000
    g = Graph("copies")
    src = g.input("data", n)
    for i in range(kernels):
        dst = g.add_storage("output" if i == kernels - 1 else "null", n)
        g.kernel(kname("fused_nn_batch_flatten", n=n), [dst, src])
        src = dst
    base = g.write(str(tmp_path), capi.plan_fn)
    s = capi.REEFScheduler(capi.REEFScheduler.REEF, 0)
    be = s.load_model_files(base + ".json", base + ".profile.json")
    rt = s.load_model_files(base + ".json", base + ".profile.json")
    s.bind_model_queue(s.create_queue(capi.REEFScheduler.BestEffortQueue), be)
    s.bind_model_queue(s.create_queue(capi.REEFScheduler.RealTimeQueue), rt)
    s.run()
    rng = np.random.default_rng(kernels)
    for i in range(12):
        x, y = rng.normal(0, 1, (2, n)).astype(np.float32)
        s.set_input(be, x)
        t = s.new_task(be)
        if i >= 4:
            s.set_input(rt, y)
            s.wait_task(s.new_task(rt))
            assert np.array_equal(s.get_output(rt), y)
        s.wait_task(t)
        assert np.array_equal(s.get_output(be), x)
    s.close()


@pytest.mark.parametrize("model", ["inception_v3_139", "densenet121_64", "resnet50_64", "bert_tiny"])
def test_branches_side_by_side(gen, model):
    """Graphs run the independent branches of a model at the same time: bit for bit what the launches in order give, for
    the graph of a whole pass and for best-effort segments."""
    base = gen(model)
    e = capi.HybridExecutor(0)
    e.load_model_from_file(base + ".json", base + ".profile.json")
    e.load_param_from_file(base + ".param")
    s = capi.REEFScheduler(capi.REEFScheduler.REEF, 0)
    mid = s.load_model_files(base + ".json", base + ".profile.json", base + ".param")
    s.bind_model_queue(s.create_queue(capi.REEFScheduler.BestEffortQueue), mid)
    s.run()
    name = "input0" if model.startswith("bert") else "data"
    rng = np.random.default_rng(5)
    for _ in range(4):
        n = e.get_data_size(name)
        x = rng.integers(0, 1000, n // 8) if name == "input0" else rng.normal(0, 1, n // 4).astype(np.float32)
        e.set_input(name, x)
        e.execute_to(e.num_kernels())
        want = e.get_output()
        e.execute_graph()
        assert np.array_equal(e.get_output(), want)
        s.set_input(mid, x, name)
        s.wait_task(s.new_task(mid))
        assert np.array_equal(s.get_output(mid), want)
    assert capi.device_error() == 0
    s.close()
    e.close()


def test_relaxed_graph_counts_its_launches():
    """The edges of a relaxed graph are indices of launches: a capture with another number of nodes than launches, or an
    edge beyond them, is refused (here on a capture of three 4-byte memsets)."""
    lib = capi.cuda_lib()
    assert lib.reef_gpu_init(C.c_int(0)) == capi.SUCC
    stream, buf = C.c_void_p(), C.c_uint64()
    assert lib.reef_stream_create(C.byref(stream), C.c_int(0)) == capi.SUCC
    assert lib.reef_malloc(C.byref(buf), C.c_size_t(12)) == capi.SUCC

    def end(launches, edges):
        assert lib.reef_graph_begin(stream) == capi.SUCC
        for i in range(3):
            assert lib.reef_memset_async(C.c_uint64(buf.value + 4 * i), C.c_int(i + 1), C.c_size_t(4), stream) == capi.SUCC
        graph = C.c_void_p()
        a, b = ((C.c_int * len(edges))(*[e[i] for e in edges]) for i in (0, 1))
        rc = lib.reef_graph_end_relaxed(stream, C.c_size_t(launches), a, b, C.c_size_t(len(edges)), C.byref(graph))
        return rc, graph

    for launches, edges, status in ((2, [(0, 1)], capi.FAIL), (4, [(0, 1), (1, 2)], capi.FAIL), (3, [(0, 3)], capi.OUT_OF_RANGE),
                                    (3, [(1, 1)], capi.OUT_OF_RANGE), (3, [(-1, 1)], capi.OUT_OF_RANGE)):
        rc, graph = end(launches, edges)
        assert rc == status and not graph.value
    rc, graph = end(3, [(0, 2)])
    assert rc == capi.SUCC and lib.reef_graph_launch(graph, stream) == capi.SUCC
    assert lib.reef_stream_sync(stream) == capi.SUCC
    got = np.zeros(12, np.uint8)
    assert lib.reef_memcpy_d2h(got.ctypes.data_as(C.c_void_p), buf, C.c_size_t(12)) == capi.SUCC
    assert got.tolist() == [1] * 4 + [2] * 4 + [3] * 4
    for rc in (lib.reef_graph_destroy(graph), lib.reef_free(buf), lib.reef_stream_destroy(stream)):
        assert rc == capi.SUCC
