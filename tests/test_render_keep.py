"""A context's kept render buffers (csrc/sms_keep.h) are given back when an
allocation would fail for them: the header's own code against a small device
(tests/render_keep_model.cpp), and no allocation of the library goes past it."""
import re
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "specular-manifold-sampling_gb300" / "csrc"


def test_kept_blocks_are_given_back(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "model"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(Path(nvcc).resolve().parents[1] / "include"),
                    "-I", str(CSRC), str(ROOT / "tests" / "render_keep_model.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout


def test_every_device_allocation_can_take_them():
    calls = {f.name: len(re.findall(r"(?<!\")\bcudaMalloc\(", f.read_text())) for f in CSRC.iterdir()
             if f.suffix in (".cu", ".cuh", ".cpp", ".h")}
    assert {n for n, k in calls.items() if k} == {"sms_keep.h"}
