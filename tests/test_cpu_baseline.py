"""The baseline of the padding throttle (csrc/host/baseline.h): samples of replays that have two speeds."""
import os
import subprocess

import pytest

from conftest import ROOT
from reef_b200 import build

MAIN = """
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "baseline.h"
int main(int argc, char** argv) {
    reef::server::ReplayBaseline b;
    for (int i = 1; i < argc; i++) {
        if (argv[i][0] == 'a') b.add_alone(atof(argv[i] + 1));
        else b.add_probe(atof(argv[i] + 1));
    }
    printf("%.17g", b.ns());
}
"""


@pytest.fixture(scope="module")
def baseline(tmp_path_factory):
    d = tmp_path_factory.mktemp("baseline")
    (d / "main.cpp").write_text(MAIN)
    subprocess.check_call([build._cxx(), "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "reef_b200", "csrc", "host"), "-o",
                           str(d / "main"), str(d / "main.cpp")])
    return lambda *samples: float(subprocess.check_output([str(d / "main")] + list(samples)))


ALONE = ["a960", "a850", "a840"] + ["a832", "a833", "a831", "a832", "a834", "a832", "a833", "a831"]


@pytest.mark.parametrize("samples,want", [
    ([], 0),                                                  # nothing measured: the scheduler falls back to the profile
    (["p806"], 806),
    (["p832", "p806", "p807", "p831"], 807),                  # two speeds: in the middle, not the least
    (["p806", "p806", "p806", "p806", "p900"], 806),          # one disturbed sample of the last four
    (["p700"] + ["p806", "p807", "p808", "p809"], 807),       # the last four count
    (ALONE, 832),                                             # cold requests left out
    (ALONE + ["p806", "p807", "p806", "p806"], 832),          # served alone before: that is what the client knows
    (ALONE[:-1] + ["p806", "p807", "p806", "p806"], 806),     # too few requests alone to go by
    (ALONE + ["p860", "p861", "p862", "p860"], 860),          # the replay has become slower since
    (ALONE + ["a700"] * 8, 700),                              # the last eight count
])
def test_baseline(baseline, samples, want):
    assert baseline(*samples) == want
