"""A best-effort task that padding left between two segment boundaries goes on by short segments; preempted inside one of them it
is resumed again.  Output: bit for bit that of an uninterrupted pass."""
import time

import numpy as np
import pytest

from conftest import seeded_input
from reef_b200 import capi

pytestmark = pytest.mark.gpu
S = capi.REEFScheduler


@pytest.mark.parametrize("model", ["resnet18_64", "inception_v3_139", "densenet121_64"])
def test_resumed_behind_padding(gen, model):
    base, rt_base = gen(model), gen("resnet18_64")
    s = S(S.REEF)
    s.run()
    rt = s.load_model_files(rt_base + ".json", rt_base + ".profile.json", rt_base + ".param")
    bes = [s.load_model_files(base + ".json", base + ".profile.json", base + ".param") for _ in range(2)]
    s.bind_model_queue(s.create_queue(S.RealTimeQueue), rt)
    for be in bes:
        s.bind_model_queue(s.create_queue(S.BestEffortQueue), be)
    n = s.get_data_size(bes[0], "data") // 4
    xs = [seeded_input(n, seed=21), seeded_input(n, seed=22)]
    s.set_input(rt, seeded_input(3 * 64 * 64, seed=15))
    want = []
    for x in xs:
        s.set_input(bes[0], x)
        s.wait_task(s.new_task(bes[0]))
        want.append(s.get_output(bes[0]))
    s.wait_task(s.new_task(rt))
    rt_want = s.get_output(rt)
    padded, resumed = 0, 0
    for i in range(40):
        time.sleep(0.03)        # no real-time request is expected any more: the window holds whole segments
        for k, be in enumerate(bes):
            s.set_input(be, xs[(i + k) % 2])
        before = s.stats()["padded_kernels"]
        tasks = [s.new_task(be) for be in bes]
        s.wait_task(s.new_task(rt))                      # pads a few kernels of either, in fours
        t0 = time.perf_counter()
        while time.perf_counter() - t0 < 10e-6 * (i % 20):
            pass
        s.wait_task(s.new_task(rt))                      # comes upon the resumed tasks
        for t in tasks:
            s.wait_task(t)
        padded += s.stats()["padded_kernels"] - before
        resumed += sum(s.get_task(t).preempted for t in tasks)
        assert np.array_equal(s.get_output(rt), rt_want)
        for k, be in enumerate(bes):
            assert np.array_equal(s.get_output(be), want[(i + k) % 2]), (i, k)
    print(model, "padded kernels", padded, "tasks preempted", resumed, "of 80")
    assert padded > 0 and resumed > 0
    assert capi.device_error() == 0
    s.shutdown()
    s.close()
