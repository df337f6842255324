"""fp32 convolution: K slices per warp (one, odd, even, none for some warps), a last slice that is not full, taps that change
inside and between slices, channels that do not fill the last tile."""
import pytest

import test_gpu_fp32_conv as fp32

pytestmark = pytest.mark.gpu

CASES = [   # ci, hi, wi, co, kh, kw, stride, ph, pw, name suffix
    (4, 5, 6, 4, 1, 1, 1, 0, 0, ""),          # a quarter of a slice; seven of eight warps without one
    (20, 7, 5, 12, 1, 1, 1, 0, 0, ""),        # a second slice of one chunk
    (12, 9, 8, 20, 3, 3, 1, 1, 1, ""),        # 6.75 slices, a tap every three chunks
    (36, 11, 7, 36, 3, 3, 2, 1, 1, ""),       # 20.25 slices, taps across slices
    (48, 13, 13, 40, 1, 7, 1, 0, 3, ""),      # 21 slices of three to a tap
    (272, 6, 6, 52, 1, 1, 1, 0, 0, ""),       # 17 slices: two or three a warp
    (512, 7, 7, 68, 3, 3, 1, 1, 1, ""),       # 288 slices: an even number for every warp
]


@pytest.mark.parametrize("case", CASES, ids=["%dx%dx%d_%d_k%dx%d" % c[:6] for c in CASES])
def test_slices_and_ragged_edges(tmp_path, case):
    """Same oracle and bound as the other shapes: fp64, against the error of a chain of fp32 multiply-adds."""
    fp32.test_fp32_convolution_against_fp64(tmp_path, case)
