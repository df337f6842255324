"""DenseNet's concatenation without elementwise kernels between the layers: the convolution that appends channels and activates
them for the next layer, and the elementwise kernel on a channel slice, against the oracle."""
import json

import numpy as np
import pytest

from conftest import rel_err
from gpu_util import TF32_TOL, all_storage, load_executor, single_kernel_model
from oracle import oracle
from reef_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,specs,written", [
    ("reef_conv2d_preact__ci128_hi7_wi7_co32_kh3_kw3_sh1_sw1_ph1_pw1_ocs160_ooff96_pcs128_poff96_v1",
     [("in", 49 * 128), ("param", 32 * 9 * 128), ("out", 49 * 160), ("param", 32), ("out", 49 * 128)], {2: (160, 96, 32), 4: (128, 96, 32)}),
    ("reef_conv2d_preact__ci32_hi5_wi9_co4_kh1_kw1_sh1_sw1_ph0_pw0_pcs8_poff4_v1",
     [("in", 45 * 32), ("param", 4 * 32), ("out", 45 * 4), ("param", 4), ("out", 45 * 8)], {2: (4, 0, 4), 4: (8, 4, 4)}),
    ("fused_add_nn_relu__c20_n63_ics40_ioff8_ocs28_ooff4", [("out", 63 * 28), ("in", 63 * 40), ("param", 20)], {0: (28, 4, 20)}),
    ("fused_add_nn_relu__c4_n1_ocs8_ooff0", [("out", 8), ("in", 4), ("param", 4)], {0: (8, 0, 4)}),
])
def test_channel_slices_against_the_oracle(tmp_path, name, specs, written):
    base, inputs = single_kernel_model(tmp_path, "one", name, specs)
    j = json.load(open(base + ".json"))
    e = load_executor(base)
    o = oracle.OracleExecutor(base + ".json", base + ".param")
    for k, v in inputs.items():
        e.set_input(k, v)
        o.set_input(k, v)
    o.execute()
    first = None
    for run in (e.execute, e.execute_preemptable, e.execute_dispatch, e.execute_graph):
        run()
        got = all_storage(e, j)
        for idx, (stride, c0, c) in written.items():
            g, w = got[idx].reshape(-1, stride), o.storage[idx].reshape(-1, stride)
            assert rel_err(g[:, c0:c0 + c], w[:, c0:c0 + c]) < TF32_TOL
            rest = np.delete(g, np.s_[c0:c0 + c], axis=1)
            assert not rest.any()            # the other channels of the buffer are left alone
        first = first or got
        assert all(np.array_equal(a, b) for a, b in zip(first, got))
    assert capi.device_error() == 0
    e.close()
