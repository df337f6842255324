"""The exchange of a K split between the ranks of a cluster, at the edges of its shares: pixel counts that are no multiple of a
group, ranks without a share, more groups than a turn takes, channels that fill no warp, both places of the receive area."""
import numpy as np
import pytest
from scipy.special import erf

from gpu_util import TF32_TOL, load_executor, single_kernel_model
from reef_b200 import capi

pytestmark = pytest.mark.gpu

CASES = [  # pixels, input channels, output channels, plan
    (1, 256, 128, "_tp16_ts8"),      # one pixel: seven ranks without a share
    (5, 256, 36, "_tp16_ts8"),       # two groups, the second ragged; channels end inside a warp
    (13, 256, 132, "_tp16_ts4"),     # four channels in the second tile
    (29, 512, 96, "_tp32_ts8"),      # the last group is one pixel
    (47, 256, 128, "_tp48_ts2"),     # six groups a half: two turns
    (64, 256, 128, "_tp64_ts4_pv1"),     # receive area over the ring
    (112, 512, 64, "_tp112_ts8"),    # the most a plan may exchange
    (128, 256, 128, "_tp128_ts2"),
    (128, 256, 128, "_tp128_ts1"),   # no split
    (300, 256, 128, "_tp112_ts2"),   # ragged last tile
]


def _model(tmp_path, name, specs, seed):
    base, inputs = single_kernel_model(tmp_path, "one", name, specs, seed=seed)
    e = load_executor(base, params=False)
    for k, v in inputs.items():
        e.set_input(k, v)
    return e, inputs


def _check(e, want):
    runs = []
    for run in (e.execute, e.execute_preemptable, e.execute_dispatch):
        run()
        runs.append(e.get_output())
        assert np.abs(runs[-1] - want).max() <= TF32_TOL * np.abs(want).max()
    assert np.array_equal(runs[0], runs[1]) and np.array_equal(runs[0], runs[2])
    assert capi.device_error() == 0


@pytest.mark.parametrize("case", CASES, ids=["%d_%d_%d%s" % c for c in CASES])
def test_shares_of_a_k_split_against_fp64(tmp_path, case):
    m, k, n, plan = case
    e, x = _model(tmp_path, f"reef_matmul_nt_bias_gelu_residual__m{m}_n{n}_k{k}_v1{plan}",
                  [("in", m * k), ("in", n * k), ("out", m * n), ("in", n), ("in", m * n)], m)
    v = x["in0"].reshape(m, k).astype(np.float64) @ x["in1"].reshape(n, k).astype(np.float64).T + x["in3"]
    _check(e, (0.5 * v * (1 + erf(v / np.sqrt(2))) + x["in4"].reshape(m, n)).ravel())
    e.close()


@pytest.mark.parametrize("case", CASES, ids=["%d_%d_%d%s" % c for c in CASES])
def test_both_outputs_of_a_k_split_against_fp64(tmp_path, case):
    m, k, n, plan = case
    e, x = _model(tmp_path, f"reef_conv2d_add_preact__ci{k}_hi1_wi{m}_co{n}_kh1_kw1_sh1_sw1_ph0_pw0_v1{plan}",
                  [("in", m * k), ("in", n * k), ("out", m * n), ("in", m * n), ("in", n), ("in", m * n)], m)
    want = (x["in0"].reshape(m, k).astype(np.float64) @ x["in1"].reshape(n, k).astype(np.float64).T + x["in3"].reshape(m, n))
    _check(e, want.ravel())
    second = e.get_data(5, 4 * m * n).reshape(m, n)
    pre = np.maximum(want + x["in4"], 0)
    assert np.abs(second - pre).max() <= TF32_TOL * np.abs(pre).max()
    e.close()

