"""The exact-fp32 attention against fp64, at the edges of its 16-row blocks, key ranges and of the line between its two forms
(148 blocks: 12 heads of 192 and 193 tokens)."""
import numpy as np
import pytest

from gpu_util import load_executor, single_kernel_model
from reef_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s,heads,mask", [(1, 1, 0), (15, 3, 0), (17, 2, 1), (128, 12, 0), (129, 12, 1), (192, 12, 0), (193, 12, 0),
                                          (250, 20, 1), (384, 12, 0), (1030, 4, 1)])
def test_attention_against_fp64(tmp_path, s, heads, mask):
    H = heads * 64
    name = f"reef_attention__s{s}_heads{heads}_d64" + ("_mask1" if mask else "")
    base, inputs = single_kernel_model(tmp_path, "one", name, [("in", s * 3 * H)] + ([("in", s)] if mask else []) + [("out", s * H)], seed=s)
    keep = np.ones(s, bool)
    if mask:
        keep = np.random.default_rng(5).random(s) > 0.3
        keep[0] = True
        inputs["in1"] = keep.astype(np.float32)
    e = load_executor(base, params=False)
    for k, v in inputs.items():
        e.set_input(k, v)
    q, k, v = inputs["in0"].astype(np.float64).reshape(s, 3, heads, 64).transpose(1, 2, 0, 3)
    sc = np.where(keep, q @ k.transpose(0, 2, 1) / 8, -np.inf)
    p = np.exp(sc - sc.max(-1, keepdims=True))
    p /= p.sum(-1, keepdims=True)
    want, size = (p @ v).transpose(1, 0, 2).ravel(), (p @ np.abs(v)).transpose(1, 0, 2).ravel()
    runs = []
    for run in (e.execute, e.execute_preemptable, e.execute_dispatch):
        run()
        runs.append(e.get_output())
    assert np.all(np.abs(runs[0] - want) <= 2e-6 * size)
    assert np.array_equal(runs[0], runs[1]) and np.array_equal(runs[0], runs[2])
    assert capi.device_error() == 0
    e.close()


@pytest.mark.parametrize("s,heads,mask", [(17, 2, 1), (128, 12, 0), (250, 20, 0)])
@pytest.mark.parametrize("where,value", [("v", np.inf), ("v", -3.4e38), ("v_last", np.inf), ("k", -np.inf), ("k", 3.4e38), ("k", np.nan), ("k_dead", np.inf)])
def test_attention_of_values_beyond_bf16(tmp_path, s, heads, mask, where, value):
    """Infinities, NaN and finite values that bf16 rounds to infinity, in one dimension of one key or value: the rows and
    columns that feel them come out as fp32 gives them (a score of -infinity is a probability of zero, +infinity NaN), the
    others within the bound above."""
    if where == "k_dead" and not mask:
        pytest.skip("needs a masked key")
    H, key, dim, head = heads * 64, s - 1 if where == "v_last" else s // 2, 37, heads - 1
    name = f"reef_attention__s{s}_heads{heads}_d64" + ("_mask1" if mask else "")
    base, inputs = single_kernel_model(tmp_path, "one", name, [("in", s * 3 * H)] + ([("in", s)] if mask else []) + [("out", s * H)], seed=s)
    keep = np.ones(s, bool)
    if mask:
        keep = np.random.default_rng(5).random(s) > 0.3
        keep[0], keep[key] = True, where != "k_dead"
        inputs["in1"] = keep.astype(np.float32)
    qkv = inputs["in0"].reshape(s, 3, heads, 64)
    qkv[:, 0, head, dim] *= 1e-3        # a finite value times the query stays finite
    qkv[key, 1 if where[0] == "k" else 2, head, dim] = value
    e = load_executor(base, params=False)
    for k, v in inputs.items():
        e.set_input(k, v)
    q, k, v = qkv.astype(np.float64).transpose(1, 2, 0, 3)
    with np.errstate(invalid="ignore"):
        sc = np.where(keep, q @ k.transpose(0, 2, 1) / 8, -np.inf)
        p = np.exp(sc - sc.max(-1, keepdims=True))
        p /= p.sum(-1, keepdims=True)
        want, size = (p @ v).transpose(1, 0, 2).ravel(), (p @ np.abs(v)).transpose(1, 0, 2).ravel()
    fin = np.isfinite(want)
    for run in (e.execute, e.execute_preemptable, e.execute_dispatch):
        run()
        got = e.get_output()
        assert np.array_equal(got[~fin], want[~fin], equal_nan=True)
        assert np.all(np.abs(got[fin] - want[fin]) <= 2e-6 * size[fin])
    assert capi.device_error() == 0
    e.close()
