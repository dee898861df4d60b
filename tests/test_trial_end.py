"""Statistics of a Bernoulli trial's end (trial_end, csrc/sms_trials.cuh), run
on the CPU: newton_iterations leaves out the trials that end past a success
that is already recorded, successful ones too."""
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_newton_iterations_of_late_trials_are_left_out(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "model"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(Path(nvcc).resolve().parents[1] / "include"),
                    "-I", str(ROOT / "specular-manifold-sampling_gb300" / "csrc"),
                    str(ROOT / "tests" / "trial_end_model.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()
    # trials 4 (fails), 5 (succeeds), then 7 and 6 past it, 2 and 3 before it, 5 past 3
    assert out[:7] == ["1", "11", "11", "11", "10011", "110011", "110011"]
    assert out[7:] == ["3", "1", "7"]   # smallest success, queries done, trials run
