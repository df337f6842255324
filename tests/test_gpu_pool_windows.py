"""Pooling windows of every form (2x2 and 3x3 read at once, other sizes tap by tap) at the borders of their input: bit for bit what
the taps give one after the other in fp32, with infinities and values below the padding's among them."""
import numpy as np
import pytest

from gpu_util import load_executor, single_kernel_model
from reef_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op,cip", [("max", 0), ("avg", 0), ("avg", 1)])
@pytest.mark.parametrize("k,s,p,hi,wi,c", [(2, 2, 0, 7, 9, 4), (2, 1, 1, 1, 5, 12), (3, 1, 1, 5, 4, 8), (3, 2, 1, 6, 7, 260), (3, 2, 0, 3, 3, 4), (4, 3, 1, 9, 8, 8)])
def test_pool_window(tmp_path, op, cip, k, s, p, hi, wi, c):
    ho, wo = (hi + 2 * p - k) // s + 1, (wi + 2 * p - k) // s + 1
    name = f"fused_nn_{op}_pool2d__c{c}_hi{hi}_wi{wi}_k{k}_s{s}_p{p}_ho{ho}_wo{wo}" + f"_cip{cip}"
    base, inputs = single_kernel_model(tmp_path, "one", name, [("in", hi * wi * c), ("out", ho * wo * c)], seed=k + c)
    x = inputs["in0"].reshape(hi, wi, c)
    if op == "max":
        x[0, 0, 0], x[-1, -1, 1], x[:, :, 2] = np.inf, -np.inf, -np.inf
    want = np.zeros((ho, wo, c), np.float32)
    for oy in range(ho):
        for ox in range(wo):
            acc, n = np.full(c, -3.402823e38 if op == "max" else 0, np.float32), 0
            for y in range(oy * s - p, oy * s - p + k):
                for q in range(ox * s - p, ox * s - p + k):
                    if 0 <= y < hi and 0 <= q < wi:
                        acc, n = np.maximum(acc, x[y, q]) if op == "max" else acc + x[y, q], n + 1
            want[oy, ox] = acc if op == "max" else acc * (np.float32(1) / np.float32(k * k if cip else max(n, 1)))
    e = load_executor(base, params=False)
    e.set_input("in0", x.ravel())
    for run in (e.execute, e.execute_preemptable, e.execute_dispatch):
        run()
        assert np.array_equal(e.get_output(), want.ravel())
    assert capi.device_error() == 0
    e.close()
