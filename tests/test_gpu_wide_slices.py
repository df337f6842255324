"""Channel slices of a buffer with more than 2^32 elements: what the tensor-core convolution stores there."""
import numpy as np
import pytest

from gpu_util import load_executor
from reef_b200 import capi
from reef_b200.resources.graph import Graph

pytestmark = pytest.mark.gpu

WIDTH, PIXELS, C = 131072, 33000, 32        # 4.3e9 elements, 17.3 GB
ONE = f"hi1_wi{PIXELS}_co{C}_kh1_kw1_sh1_sw1_ph0_pw0"


@pytest.mark.parametrize("flavour", ["execute", "execute_preemptable"])
def test_both_outputs_beyond_2_to_the_32_elements(tmp_path, flavour):
    """Weights are the identity and every value has ten mantissa bits, so both slices come back exactly."""
    rng = np.random.default_rng(3)
    x = rng.integers(-512, 513, PIXELS * C).astype(np.float32)
    bias = rng.integers(-64, 65, C).astype(np.float32)
    g = Graph("wide")
    xi = g.input("in0", PIXELS * C)
    eye, b = g.param(np.eye(C, dtype=np.float32)), g.param(bias)
    wide = g.add_storage("temp", WIDTH * PIXELS)
    outs = [g.add_storage("output", PIXELS * C) for _ in range(2)]
    g.kernel(f"reef_conv2d_preact__ci{C}_{ONE}_ocs{WIDTH}_ooff{WIDTH - C}_pcs{WIDTH}_poff64_v1", [xi, eye, wide, b, wide])
    for out, off in zip(outs, (WIDTH - C, 64)):
        g.kernel(f"fused_nn_conv2d__ci{C}_{ONE}_ics{WIDTH}_ioff{off}_v1", [wide, eye, out])
    base = g.write(str(tmp_path), capi.plan_fn)
    e = load_executor(base)
    e.set_input("in0", x)
    getattr(e, flavour)()
    first, second = (e.get_data(o, 4 * PIXELS * C) for o in outs)
    assert np.array_equal(first, x)
    assert np.array_equal(second, np.maximum(x.reshape(PIXELS, C) + bias, 0).ravel())
    assert capi.device_error() == 0
    e.close()
