"""The FP32 path's jumps (newman_gb300/csrc/jump.hpp) against the iterations they
stand for: the polynomial of a record within its bound of the exact orbit and of
the plain FP64 path's own steps, from the series stop and from a rebase (the
FP64 path at the same orbit index and left at another after a near return), with
no bailout and no rebase on the way.  Long double on the host
(tests/native/jump_check.cpp); the device evaluates the same records.  CPU only."""
import json
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "newman_gb300", "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
WALK = json.load(open(os.path.join(HERE, "golden", "deep_centers.json")))["steps"]
SEAHORSE = ("-0.743643887037151", "0.131825904205330")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("jump") / "jump_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-pthread", "-I", CSRC,
                    "-I", os.path.join(ROOT, "include"), "-I", CUDA_INC,
                    os.path.join(HERE, "native", "jump_check.cpp"),
                    os.path.join(CSRC, "jump.cpp"), os.path.join(CSRC, "mpview.cpp"),
                    "-o", exe, "-l:libgmp.so.10"], check=True)
    return exe


def center(width_exp):
    k = next(i for i, s in enumerate(WALK) if float(s["width"]) <= 10.0 ** -width_exp)
    return WALK[k - 1]["next_center_re"], WALK[k - 1]["next_center_im"]


# (center, step, rows, cols, N, reference): the largest relative eps (1e-12), the
# probe and the center orbit, eps below the orders kept, ragged and tiny grids,
# floatexp tables
@pytest.mark.parametrize("where,step,nr,nc,N,mode", [
    (SEAHORSE, "1.302083e-16", 540, 960, 50000, "probes"),
    (SEAHORSE, "1e-16", 201, 333, 50000, "probes"),
    (SEAHORSE, "1e-17", 37, 65, 50000, "center"),
    (16, "2e-19", 97, 131, 20000, "center"),
    (40, "1e-43", 61, 83, 60000, "center"),
    (160, "1e-163", 48, 64, 130000, "center"),
])
def test_jumps_stay_within_their_bounds(check, where, step, nr, nc, N, mode):
    re, im = where if isinstance(where, tuple) else center(where)
    out = subprocess.run([check, re, im, step, str(nr), str(nc), str(N), mode, "400", "9"],
                         capture_output=True, text=True)
    rebases, starts = [line.split() for line in out.stdout.strip().splitlines()]
    assert out.returncode == 0 and rebases[1] == "0" and starts[2] == "0", out.stdout
    assert int(rebases[0]) > 100 and float(rebases[2]) > 16  # jumps were made, and far
