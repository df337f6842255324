"""A K split of which one rank waits for a load that never comes: the launch ends by itself, with the error word set and nobody's
shared memory left behind while a peer could still store into it, and the next launches are as good as any."""
import ctypes as C
import glob
import os

import numpy as np
import pytest

from gpu_util import TF32_TOL
from reef_b200 import build

HERE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")
LIMIT_MS = 50


def _library():
    src, out = os.path.join(HERE, "exchange_timeout.cu"), os.path.join(HERE, "libexchange_timeout.so")
    deps = [src] + glob.glob(os.path.join(build.CSRC, "kernels", "*")) + glob.glob(os.path.join(build.INCLUDE, "*.h"))
    build._build(out, [build._nvcc()] + build.NVCC_FLAGS + ["-DREEF_DEBUG_AIDS", f"-DREEF_WAIT_LIMIT_NS={LIMIT_MS}000000ull", "-I", build.INCLUDE, "-o", out, src],
                 deps, False)
    return out


def test_the_limited_build_compiles():
    assert os.path.exists(_library())


CASES = [  # pixels, output channels, K, tile cap, ranks, rank that waits, its K block
    (64, 128, 1024, 64, 8, 3, 3),       # four K blocks a rank: a load of the first fill, the last one
    (64, 128, 1024, 64, 8, 0, 0),       # the first one, of a rank whose peers' stores come earliest
    (28, 132, 4096, 32, 8, 7, 14),      # a refill
    (5, 256, 256, 16, 8, 5, 0),         # ranks without a share wait for nobody, the one that gives up stores to others
    (112, 128, 2304, 112, 4, 1, 17),    # the receive area lies over the ring
    (128, 128, 512, 128, 2, 1, 7),
    (128, 128, 512, 128, 1, 0, 15),     # no split
]


@pytest.mark.gpu
@pytest.mark.parametrize("delay", [0, 2 * LIMIT_MS])      # in the second case the peers give up long before its shares come
@pytest.mark.parametrize("best_effort", [0, 1])
@pytest.mark.parametrize("case", CASES, ids=["%d_%d_%d_ts%d_rank%d_load%d" % (c[:3] + c[4:]) for c in CASES])
def test_a_wait_of_the_exchange_that_expires(case, best_effort, delay):
    m, n, k, cap, splits, rank, load = case
    lib = C.CDLL(_library())
    rng = np.random.default_rng(m)
    x, w = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((n, k), dtype=np.float32)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    f32 = lambda a: a.ctypes.data_as(C.POINTER(C.c_float))      # noqa: E731

    def run(rank, load, delay=0):
        out, plan, slot, error, ms = np.zeros((m, n), np.float32), (C.c_int * 4)(), C.c_int(), C.c_int(), C.c_float()
        rc = lib.exchange_run(m, n, k, cap, splits, best_effort, rank, load, delay, f32(x), f32(w), f32(out), plan, C.byref(slot), C.byref(error), C.byref(ms))
        assert rc == 0
        return out, list(plan), slot.value, error.value, ms.value

    def good():
        out, (ranks, tiles, blocks, _), slot, error, _ = run(-1, -1)
        assert ranks == splits and load < blocks
        assert error == 0 and slot == ranks * tiles
        assert np.abs(out - want).max() <= TF32_TOL * np.abs(want).max()
        return out

    before = good()
    _, (ranks, tiles, _, over_ring), slot, error, ms = run(rank, load, delay)
    print(case, "best-effort" if best_effort else "plain", f"ended after {ms:.1f} ms, {slot} of {ranks * tiles} CTAs complete")
    assert error == 1
    groups = -(-min(m, cap) // 4)
    receivers = -(-groups // -(-groups // ranks))      # ranks with a share
    # CTAs that cannot have counted themselves complete when it comes too late (over the ring, a barrier holds all ranks until it does)
    late = receivers + (rank >= receivers) if delay and not over_ring else 1
    assert slot <= ranks * tiles - late
    # the wait that expires, the peers' shares and the own loads, each with a limit of its own
    assert LIMIT_MS + delay <= ms <= 3.5 * LIMIT_MS + delay
    for _ in range(3):
        assert np.array_equal(good(), before)
