"""The host sources compile for hosts without x86 intrinsics (an Arm host of a GPU has none)."""
import glob
import os
import subprocess

import pytest

from conftest import ROOT
from reef_b200 import build

HOST = os.path.join(ROOT, "reef_b200", "csrc", "host")


@pytest.mark.parametrize("source", sorted(os.path.basename(p) for p in glob.glob(os.path.join(HOST, "*.cpp"))))
def test_host_source_without_x86_intrinsics(tmp_path, source):
    for header in ("emmintrin.h", "immintrin.h", "xmmintrin.h", "x86intrin.h"):
        (tmp_path / header).write_text("#error an x86 header on a host that is not x86\n")
    subprocess.check_call([build._cxx(), "-std=c++17", "-fsyntax-only", "-Wall", "-Werror", "-U__SSE2__", "-I", str(tmp_path),
                           "-I", os.path.join(ROOT, "include"), os.path.join(HOST, source)])
