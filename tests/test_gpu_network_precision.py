"""Whole TF32 networks against the same schedule in fp64: what reaches the softmax (or, for an encoder, the output) in 2-norm.

Bound: every kernel rounds the activations that it stores to 11 significant bits.  The error of one rounding is uniform in
+- 2^-11 of the leading bit, 2^-11 / sqrt(3) x 0.74 = 0.42 x 2^-11 of the value in the mean square over a mantissa; the roundings
of a schedule's kernels add as independent ones, no more than all of them along one path: 0.42 x 2^-11 x sqrt(kernels)."""
import json

import numpy as np
import pytest

from gpu_util import load_executor
from oracle.torch_ref import TorchExecutor
from reef_b200 import capi

pytestmark = pytest.mark.gpu

MODELS = [("resnet18", dict(image=64)), ("resnet50", dict(image=97)), ("inception_v3", dict(image=139)), ("densenet201", dict(image=64)),
          ("vgg16_32", {}), ("bert_base", dict(layers=2, hidden=128, heads=2, ffn=256, vocab=1000, seq=77))]


@pytest.mark.parametrize("model,kw", MODELS, ids=[m for m, _ in MODELS])
def test_network_against_fp64(gen, tmp_path, model, kw):
    from reef_b200 import resources
    base = f"{resources.generate(model, str(tmp_path), **kw)}/{model}"
    j = json.load(open(base + ".json"))
    data = j["storage"][0]
    rng = np.random.default_rng(16)
    x = rng.integers(0, 1000, data["size"]).astype(np.int64) if data["stype"] == "int64" else rng.normal(0, 1, data["size"]).astype(np.float32)
    e, o = load_executor(base), TorchExecutor(base + ".json", base + ".param", double=True)
    for ref in (e, o):
        ref.set_input(data["name"], x)
        ref.execute()
    last = j["kernels"][-1]
    at = last["args"][0]        # a softmax's argument, or the output of an encoder's last LayerNorm
    want = o.t[at].numpy().ravel()
    err = np.linalg.norm(e.get_data(at, 4 * want.size) - want) / np.linalg.norm(want)
    bound = 0.42 * 2.0 ** -11 * len(j["kernels"]) ** 0.5
    print(f"{model}: {err:.2e}, bound {bound:.2e}")
    assert err <= bound
    assert capi.device_error() == 0
    e.close()
