"""The exact-fp32 convolution (operands split into bf16 values on the tensor cores): against fp64, at the edges of its tiles,
K slices and loaders.  The error bound is that of a chain of fp32 multiply-adds, scaled by the size of the sum."""
import numpy as np
import pytest
import torch

from gpu_util import load_executor, single_kernel_model
from reef_b200 import capi

pytestmark = pytest.mark.gpu

CASES = [  # ci, hi, wi, co, kh, kw, s, ph, pw, extra
    (256, 13, 13, 256, 3, 3, 1, 1, 1, ""),        # eight warps share a tile's K
    (64, 49, 49, 64, 3, 3, 1, 1, 1, ""),
    (64, 17, 31, 256, 1, 1, 1, 0, 0, ""),         # two slices of K
    (512, 7, 7, 36, 3, 3, 2, 1, 1, ""),           # 16 pixels, channels end inside a tile
    (4, 5, 3, 4, 1, 1, 1, 0, 0, ""),              # less than one slice, one pixel tile
    (20, 9, 9, 12, 1, 7, 1, 0, 3, ""),            # chunks of one slice in several taps
    (48, 1, 1, 8, 5, 5, 1, 2, 2, ""),             # one pixel, every tap but one in the padding
    (3, 37, 41, 64, 7, 7, 2, 3, 3, "_nchw1"),     # planar input
    (6, 11, 10, 20, 3, 3, 1, 1, 1, ""),           # channel count without 16-byte chunks
    (8, 40, 3, 8, 33, 1, 1, 16, 0, ""),           # more filter rows than a mask has bits
]


@pytest.mark.parametrize("case", CASES, ids=["%dx%dx%d_%d_k%dx%d%s" % (c[:6] + (c[9],)) for c in CASES])
def test_fp32_convolution_against_fp64(tmp_path, case):
    ci, hi, wi, co, kh, kw, s, ph, pw, extra = case
    ho, wo = (hi + 2 * ph - kh) // s + 1, (wi + 2 * pw - kw) // s + 1
    name = f"fused_nn_conv2d_add__ci{ci}_hi{hi}_wi{wi}_co{co}_kh{kh}_kw{kw}_sh{s}_sw{s}_ph{ph}_pw{pw}{extra}"
    specs = [("in", ci * hi * wi), ("param", co * kh * kw * ci), ("out", ho * wo * co), ("in", ho * wo * co)]
    base, inputs = single_kernel_model(tmp_path, "one", name, specs, seed=ci)
    e = load_executor(base)
    for k, v in inputs.items():
        e.set_input(k, v)
    x = torch.from_numpy(inputs["in0"]).double()
    x = x.view(1, ci, hi, wi) if extra else x.view(1, hi, wi, ci).permute(0, 3, 1, 2)
    w = torch.from_numpy(e.get_data(1, 4 * co * kh * kw * ci)).double().view(co, kh, kw, ci).permute(0, 3, 1, 2)
    res = torch.from_numpy(inputs["in3"]).double().view(ho, wo, co)
    conv = lambda a, b: torch.nn.functional.conv2d(a, b, stride=s, padding=(ph, pw))[0].permute(1, 2, 0)   # noqa: E731
    want, size = (conv(x, w) + res).numpy().ravel(), (conv(x.abs(), w.abs()) + res.abs()).numpy().ravel()
    runs = []
    for run in (e.execute, e.execute_preemptable, e.execute_dispatch):
        run()
        runs.append(e.get_output())
        assert np.all(np.abs(runs[-1] - want) <= 3e-7 * size)
    assert np.array_equal(runs[0], runs[1]) and np.array_equal(runs[0], runs[2])
    assert capi.device_error() == 0
    e.close()


def _as_fp32(want):
    """What fp32 makes of fp64 results: beyond its largest value, infinity."""
    return np.where(np.abs(want) > np.finfo(np.float32).max, np.copysign(np.inf, want), want)


@pytest.mark.parametrize("case", [CASES[i] for i in (0, 2, 5, 7, 8)], ids=["%dx%dx%d_%d_k%dx%d%s" % (CASES[i][:6] + (CASES[i][9],)) for i in (0, 2, 5, 7, 8)])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.4e38, -3.397e38])
def test_fp32_convolution_of_values_beyond_bf16(tmp_path, case, value):
    """Infinities, NaN and finite values that bf16 rounds to infinity: as fp32 multiply-adds give them, where they are felt
    (one pixel, so that no two of them meet in a sum) and nowhere else.  Same bound as above elsewhere."""
    ci, hi, wi, co, kh, kw, s, ph, pw, extra = case
    ho, wo = (hi + 2 * ph - kh) // s + 1, (wi + 2 * pw - kw) // s + 1
    name = f"fused_nn_conv2d__ci{ci}_hi{hi}_wi{wi}_co{co}_kh{kh}_kw{kw}_sh{s}_sw{s}_ph{ph}_pw{pw}{extra}"
    base, inputs = single_kernel_model(tmp_path, "one", name, [("in", ci * hi * wi), ("param", co * kh * kw * ci), ("out", ho * wo * co)], seed=ci)
    e = load_executor(base)
    x = inputs["in0"].reshape((ci, hi, wi) if extra else (hi, wi, ci))
    x[(ci // 2, hi // 2, wi // 2) if extra else (hi // 2, wi // 2, ci // 2)] = value
    e.set_input("in0", inputs["in0"])
    x = torch.from_numpy(x).double()
    x = (x if extra else x.permute(2, 0, 1)).unsqueeze(0)
    w = torch.from_numpy(e.get_data(1, 4 * co * kh * kw * ci)).double().view(co, kh, kw, ci).permute(0, 3, 1, 2)
    conv = lambda a, b: torch.nn.functional.conv2d(a, b, stride=s, padding=(ph, pw))[0].permute(1, 2, 0).numpy().ravel()   # noqa: E731
    want, size = _as_fp32(conv(x, w)), conv(x.abs(), w.abs())
    fin = np.isfinite(want)
    assert 0 < (~np.isfinite(size)).sum() < want.size or abs(value) < 3.5e38
    for run in (e.execute, e.execute_preemptable, e.execute_dispatch):
        run()
        got = e.get_output()
        assert np.array_equal(got[~fin], want[~fin], equal_nan=True)
        assert np.all(np.abs(got[fin] - want[fin]) <= 3e-7 * size[fin])
    assert capi.device_error() == 0
    e.close()
