"""Completion counters of a preempted run: a kernel behind one that left early may run whole, over partial data, and have a full
counter.  The run is resumed from the first short counter all the same."""
import numpy as np
import pytest

from gpu_util import load_executor
from reef_b200 import capi
from reef_b200.resources.graph import Graph

pytestmark = pytest.mark.gpu

# behind a GEMV of 411 MB (70 us, polls at each refill of its ring): kernels without polls, resident early
TAILS = {
    "softmax": ("fused_nn_softmax__rows1_n4096", 4096),
    "add_relu": ("fused_add_nn_relu__c4096_n1", 4096),
}


@pytest.mark.parametrize("tail", list(TAILS))
def test_a_full_counter_behind_a_short_one_is_not_trusted(tmp_path, tail):
    name, n = TAILS[tail]
    rng = np.random.default_rng(9)
    g = Graph("tail")
    x = g.input("in0", 25088)
    w = g.param(rng.standard_normal(4096 * 25088, dtype=np.float32) * 0.01)
    b = g.param(rng.standard_normal(4096, dtype=np.float32))
    mid, out = g.add_storage("temp", 4096), g.add_storage("output", n)
    g.kernel("fused_nn_dense_add__k25088_n4096", [x, w, mid, b])
    g.kernel(name, [mid, out] if tail == "softmax" else [mid, b, out])
    base = g.write(str(tmp_path), capi.plan_fn)
    e = load_executor(base)
    inputs = [rng.standard_normal(25088, dtype=np.float32) for _ in range(2)]
    want = []
    for v in inputs:
        e.set_input("in0", v)
        e.execute_preemptable()
        want.append(e.get_output())
    blocks = e.task_slots()[1]
    trusted_would_be_wrong = 0
    for i in range(60):
        e.set_input("in0", inputs[i % 2])     # (the other input's results are in the buffers)
        restarts, first = e.execute_preempt_resume(10 + i)
        assert np.array_equal(e.get_output(), want[i % 2]), f"delay {10 + i} us: {restarts} restarts from kernel {first}"
        found = e.preempted_slots()
        trusted_would_be_wrong += restarts > 0 and found[0] < blocks[0] and found[1] == blocks[1]
    print(tail, "full behind a short one in", trusted_would_be_wrong, "of 60 runs")
    assert trusted_would_be_wrong > 0
    assert capi.device_error() == 0
    e.close()
