"""The FP64 step's FP32 estimates that spare Y, |Y|^2 and |delta|^2, and the eps it
leaves out (newman_gb300/csrc/pixel_fp64.cuh), against the FP64 operations they
stand for: no mismatch (tests/native/fp64_estimate.cpp).  CPU only."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.mark.parametrize("seed", [3, 77])
def test_estimates_agree_with_fp64(tmp_path, seed):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = str(tmp_path / "fp64_estimate")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    "-I", os.path.join(ROOT, "newman_gb300", "csrc"), "-I", CUDA_INC,
                    os.path.join(HERE, "native", "fp64_estimate.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe, "2000000", str(seed)], capture_output=True, text=True)
    words = out.stdout.split()
    assert out.returncode == 0 and words[-2] == "0", out.stdout
    assert int(words[2]) > 100000 and int(words[4]) > 10000  # both were exercised
