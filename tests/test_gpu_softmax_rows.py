"""Softmax of a row kept in registers and of a longer one read three times: both sides of the limit, and the smallest row; dense
layers whose rows end inside a piece or a block's first fill."""
import numpy as np
import pytest

from gpu_util import load_executor, single_kernel_model
from reef_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 1000, 2047, 2048, 2049, 5000])
def test_softmax_row_lengths(tmp_path, n):
    base, inputs = single_kernel_model(tmp_path, "one", f"fused_nn_softmax__n{n}", [("in", n), ("out", n)], seed=n)
    e = load_executor(base, params=False)
    x = inputs["in0"] * 8
    e.set_input("in0", x)
    e.execute()
    got = e.get_output()
    w = np.exp(x.astype(np.float64) - x.max())
    assert np.abs(got - w / w.sum()).max() <= 1e-6
    e.execute_preemptable()
    assert np.array_equal(e.get_output(), got)
    e.close()


@pytest.mark.parametrize("k,n", [(4, 1), (2052, 300), (4096, 37), (6, 9)])
def test_dense_row_ends(tmp_path, k, n):
    base, inputs = single_kernel_model(tmp_path, "one", f"fused_nn_dense_add__k{k}_n{n}", [("in", k), ("param", n * k), ("out", n), ("param", n)], seed=k)
    e = load_executor(base)
    e.set_input("in0", inputs["in0"])
    w, b = (e.get_data(i, 4 * s).astype(np.float64) for i, s in ((1, n * k), (3, n)))
    want = w.reshape(n, k) @ inputs["in0"].astype(np.float64) + b
    for run in (e.execute, e.execute_graph, e.execute_preemptable):
        run()
        assert np.abs(e.get_output() - want).max() <= 1e-5 * np.abs(want).max() + 1e-6
    assert capi.device_error() == 0
    e.close()
