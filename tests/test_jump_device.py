"""The FP32 path's jumps as the device makes them (newman_gb300/csrc/fe_jump.cuh in
its host build, tests/native/jump_device.cpp) against the records' polynomials in
long double.  CPU only."""
import os
import shutil
import subprocess

import pytest

from test_jumps import CSRC, CUDA_INC, HERE, ROOT, SEAHORSE, center


def compiled(tmp_path_factory, name):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp(name) / name)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-pthread", "-I", CSRC,
                    "-I", os.path.join(ROOT, "include"), "-I", CUDA_INC,
                    os.path.join(HERE, "native", name + ".cpp"),
                    os.path.join(CSRC, "jump.cpp"), os.path.join(CSRC, "mpview.cpp"),
                    "-o", exe, "-l:libgmp.so.10", "-ldl"], check=True)
    return exe


@pytest.fixture(scope="module")
def threads(tmp_path_factory):
    return compiled(tmp_path_factory, "jump_threads")


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    exe = compiled(tmp_path_factory, "jump_device")

    def go(what, where, step, nr, nc, N, mode, samples=20000, seed=5):
        re, im = where if isinstance(where, tuple) else center(where)
        out = subprocess.run([exe, what, re, im, step, str(nr), str(nc), str(N), mode,
                              str(samples), str(seed)], capture_output=True, text=True)
        assert out.returncode in (0, 1) and out.stdout, out.stderr
        return out.stdout.split()
    return go


# The whole grid of a 1920x1080x16 view (the largest eps beside the balls), both
# references; eps small beside most balls; eps below the orders kept.
@pytest.mark.parametrize("where,step,nr,nc,N,mode", [
    (SEAHORSE, "1.302083e-16", 4320, 7680, 50000, "probes"),
    (SEAHORSE, "1.302083e-16", 4320, 7680, 50000, "center"),
    (18, "1e-18", 541, 961, 50000, "center"),
    (40, "1e-43", 61, 83, 60000, "center"),
])
def test_bound_grows_by_the_whole_derivative(run, where, step, nr, nc, N, mode):
    jumps, bad, worst = run("slope", where, step, nr, nc, N, mode)
    assert bad == "0" and int(jumps) > 3000, (jumps, bad, worst)


# One component of eps exactly 0: the row and the column of a view-center reference.
@pytest.mark.parametrize("where,step,nr,nc,N,mode", [
    (SEAHORSE, "1e-17", 37, 65, 50000, "center"),
    (18, "1e-18", 541, 961, 50000, "center"),
    (160, "1e-163", 48, 64, 130000, "center"),
])
def test_start_jumps_on_the_axes(run, where, step, nr, nc, N, mode):
    jumps, bad, worst = run("start", where, step, nr, nc, N, mode)
    assert bad == "0" and int(jumps) > 1000, (jumps, bad, worst)


# eps beyond the grid that the tables were built for, by 2^-20 to 2 times.
@pytest.mark.parametrize("where,step,nr,nc,N,mode", [
    (SEAHORSE, "1e-17", 37, 65, 50000, "center"),
    (18, "1e-18", 541, 961, 50000, "center"),
])
def test_no_chain_jump_beyond_the_grid(run, where, step, nr, nc, N, mode):
    inside, beyond, part = run("range", where, step, nr, nc, N, mode)
    assert beyond == "0" and int(inside) > 500 and float(part) > 0.5, (inside, beyond, part)


def test_ties_of_the_rebase_test_at_every_size(run):
    samples, bad, _ = run("tie", SEAHORSE, "1e-17", 37, 65, 1000, "center")
    assert bad == "0", bad


def test_side_of_a_tie_is_the_fp64_path_s(run):
    ties, bad, decided = run("side", SEAHORSE, "1e-17", 37, 65, 1000, "center", samples=2000000)
    assert bad == "0" and int(ties) > 10000 and float(decided) > 0.5, (ties, bad, decided)


# (eps above the float range: the float-float steps hold it unscaled)
@pytest.mark.parametrize("where,step,nr,nc,N,mode", [
    (SEAHORSE, "1.302083e-16", 4320, 7680, 50000, "probes"),
    (SEAHORSE, "3e-17", 97, 131, 50000, "center"),
    (17, "2e-20", 97, 131, 20000, "center"),
    (20, "1e-23", 97, 131, 50000, "center"),
    (25, "1e-28", 97, 131, 40000, "center"),
    (28, "1e-31", 97, 131, 40000, "center"),
])
def test_jumps_are_as_near_as_the_steps(run, where, step, nr, nc, N, mode):
    jumps, bad, worst = run("precision", where, step, nr, nc, N, mode, samples=1500)
    assert bad == "0" and int(jumps) > 300, (jumps, bad, worst)


@pytest.mark.parametrize("where,step,N", [(SEAHORSE, "1e-16", 50000), (20, "1e-22", 20000),
                                          (40, "1e-43", 60000)])
def test_tables_keep_to_their_threads(threads, where, step, N):
    re, im = where if isinstance(where, tuple) else center(where)
    out = subprocess.run([threads, re, im, step, "97", "131", str(N)], capture_output=True,
                         text=True)
    differ, beyond, started = out.stdout.split()
    assert differ == "0" and beyond == "0" and int(started) > 0, out.stdout


# (center, step, N, grids of 2^17 - 1, 2^17, 499,999 and 500,000 samples with tables):
# long start jumps; short ones; none, a center known to 15 digits far below them
@pytest.mark.parametrize("where,step,N,tables", [
    (25, "2e-28", 40000, "0111"),
    (SEAHORSE, "2e-17", 50000, "0001"),
    (SEAHORSE, "1e-28", 60000, "0000"),
])
def test_tables_only_where_they_pay(run, where, step, N, tables):
    assert run("sizes", where, step, 333, 517, N, "center")[0] == tables
