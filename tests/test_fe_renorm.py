"""The FE32 path's scaled steps (newman_gb300/csrc/fe_core.cuh) give the same state,
bit for bit, in whatever pieces a warp makes them: the exponent is set after every
NM_OPT_RENORM steps of the sample (tests/native/fe_renorm.cpp).  CPU only."""
import json
import os
import shutil
import subprocess
from decimal import Decimal

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "newman_gb300", "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
WALK = json.load(open(os.path.join(HERE, "golden", "deep_centers.json")))["steps"]


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    path = str(tmp_path_factory.mktemp("renorm") / "fe_renorm")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-pthread", "-I", CSRC,
                    "-I", os.path.join(ROOT, "include"), "-I", CUDA_INC,
                    os.path.join(HERE, "native", "fe_renorm.cpp"),
                    os.path.join(CSRC, "mpview.cpp"), "-o", path, "-l:libgmp.so.10"], check=True)
    return path


@pytest.mark.parametrize("width,step", [("1e-30", "1e-31"), ("1e-45", "1e-47")])
def test_pieces_do_not_change_the_state(exe, width, step):
    at = WALK[next(i for i, s in enumerate(WALK) if Decimal(s["width"]) <= Decimal(width)) - 1]
    out = subprocess.run([exe, at["next_center_re"], at["next_center_im"], step, "48", "64",
                          "20000", "400", "19990", "3"], capture_output=True, text=True)
    samples, mismatches, renormalisations = out.stdout.split()
    assert out.returncode == 0 and mismatches == "0", out.stdout
    assert int(renormalisations) > 400  # more than one a sample: pieces were cut
