"""The tensor-core convolution cut into tiles: rows in ragged pieces, ragged groups of rows, and the plans that the cost model
picks at the edges of its range, against fp64."""
import numpy as np
import pytest
import torch

from gpu_util import TF32_TOL, load_executor, single_kernel_model
from reef_b200 import capi

pytestmark = pytest.mark.gpu

CASES = [  # ci, hi, wi, co, kh, kw, s, ph, pw, plan in the name
    (64, 5, 37, 132, 3, 3, 1, 1, 1, "_tp16_ts1"),    # rows of 37 as 13 + 13 + 11
    (64, 3, 229, 64, 3, 3, 1, 1, 1, "_tp208_ts4"),   # 115 + 114, K split
    (32, 4, 45, 64, 1, 7, 2, 0, 3, "_tp8_ts2"),      # 8 + 8 + 7 from a strided input
    (64, 7, 7, 128, 3, 3, 1, 1, 1, "_tp48_ts8"),     # 7 rows as 4 + 3
    (64, 17, 17, 64, 3, 3, 1, 1, 1, "_tp64_ts2"),    # five groups of 3 rows and one of 2
    (32, 3, 211, 64, 3, 3, 1, 1, 1, ""),             # no divisor at all: the cost model's choice
    (32, 1, 1, 4, 1, 1, 1, 0, 0, ""),                # one pixel
    (2048, 4, 4, 384, 1, 1, 1, 0, 0, ""),            # all of K, few pixels
]


@pytest.mark.parametrize("case", CASES, ids=["%dx%dx%d_%d_k%dx%d%s" % (c[:6] + (c[9],)) for c in CASES])
def test_tensor_core_tiles_against_fp64(tmp_path, case):
    ci, hi, wi, co, kh, kw, s, ph, pw, plan = case
    ho, wo = (hi + 2 * ph - kh) // s + 1, (wi + 2 * pw - kw) // s + 1
    name = f"fused_nn_conv2d_add__ci{ci}_hi{hi}_wi{wi}_co{co}_kh{kh}_kw{kw}_sh{s}_sw{s}_ph{ph}_pw{pw}_v1{plan}"
    specs = [("in", ci * hi * wi), ("param", co * kh * kw * ci), ("out", ho * wo * co), ("in", ho * wo * co)]
    base, inputs = single_kernel_model(tmp_path, "one", name, specs, seed=ci)
    e = load_executor(base)
    for k, v in inputs.items():
        e.set_input(k, v)
    x = torch.from_numpy(inputs["in0"]).double().view(1, hi, wi, ci).permute(0, 3, 1, 2)
    w = torch.from_numpy(e.get_data(1, 4 * co * kh * kw * ci)).double().view(co, kh, kw, ci).permute(0, 3, 1, 2)
    want = torch.nn.functional.conv2d(x, w, stride=s, padding=(ph, pw))[0].permute(1, 2, 0).numpy().ravel() + inputs["in3"]
    runs = []
    for run in (e.execute, e.execute_preemptable, e.execute_dispatch):
        run()
        runs.append(e.get_output())
        assert np.abs(runs[-1] - want).max() <= TF32_TOL * np.abs(want).max()
    assert np.array_equal(runs[0], runs[1]) and np.array_equal(runs[0], runs[2])
    assert capi.device_error() == 0
    e.close()
