"""The Bernoulli trials' stream (csrc/sms_trials.cuh) on the CPU: its own code
under randomly drawn interleavings of its warps (tests/trial_stream_model.cpp).
Whatever the order, a query's count is its smallest successful trial
(manifold_ss.cpp:115-135)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path_factory.mktemp("trials") / "model"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(Path(nvcc).resolve().parents[1] / "include"),
                    "-I", str(ROOT / "specular-manifold-sampling_gb300" / "csrc"),
                    str(ROOT / "tests" / "trial_stream_model.cpp"), "-o", str(exe)], check=True)
    return exe


# (runs, warps, queries, cap, percent of trials that succeed, claim size):
# one query and few warps, a claim of several trials, lists that end together,
# and (40 of 64 lanes, 64 trials) a list whose first trials run in a pass of their own
@pytest.mark.parametrize("case", [(2000, 2, 1, 4, 60, 1), (2000, 3, 2, 6, 50, 1), (2000, 4, 3, 8, 40, 2),
                                  (500, 8, 5, 16, 30, 1), (300, 2, 40, 64, 20, 1)])
def test_smallest_successful_trial_whatever_the_order(model, case):
    r = subprocess.run([str(model), *map(str, case)], capture_output=True, text=True, timeout=120, check=True)
    assert int(r.stdout) == 0
