"""LayerNorm with a row divided among warps, against fp64: every number of warps to a row, ragged widths and row counts, and the
division into blocks that schedules of earlier versions state."""
import numpy as np
import pytest

from gpu_util import load_executor, single_kernel_model
from reef_b200 import capi

pytestmark = pytest.mark.gpu

# A result is ((x - mean) * rstd) * gamma + beta in fp32: five roundings of values up to |gamma| * 4 sigma and the errors of two
# sums of h terms, each at most log2(h) + 2 roundings deep: below 20 eps of the largest result.
TOL = 20 * 2.0 ** -24


@pytest.mark.parametrize("h", [128, 256, 384, 512, 640, 768, 1024])
@pytest.mark.parametrize("rows,res,suffix", [(1, 0, ""), (3, 1, ""), (17, 1, ""), (9, 0, "_pv1"), (131, 1, "_pv1")])
def test_layernorm_against_fp64(tmp_path, h, rows, res, suffix):
    name = f"reef_{'add_' if res else ''}layernorm__rows{rows}_h{h}{suffix}"
    specs = [("out", rows * h)] + [("in", rows * h)] * (1 + res) + [("in", h)] * 2
    base, x = single_kernel_model(tmp_path, "one", name, specs, seed=h + rows)
    e = load_executor(base, params=False)
    for k, v in x.items():
        e.set_input(k, v)
    d = {int(k[2:]): v.astype(np.float64) for k, v in x.items()}
    v = d[1].reshape(rows, h) + (d[2].reshape(rows, h) if res else 0)
    v = (v - v.mean(1, keepdims=True)) / np.sqrt(v.var(1, keepdims=True) + 1e-12)
    want = (v * d[2 + res] + d[3 + res]).ravel()
    runs = []
    for run in (e.execute, e.execute_preemptable, e.execute_dispatch):
        run()
        runs.append(e.get_output())
        assert np.abs(runs[-1] - want).max() <= TOL * np.abs(want).max()
    assert np.array_equal(runs[0], runs[1]) and np.array_equal(runs[0], runs[2])
    assert capi.device_error() == 0
    e.close()
