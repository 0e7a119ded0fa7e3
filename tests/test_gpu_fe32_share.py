"""Which samples the FE32 path leaves to the FP64 kernel, and how near its smoothing
stays to that kernel's."""
import numpy as np
import pytest

from helpers import C2, setup_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nm():
    import newman_gb300
    newman_gb300.load_library()
    return newman_gb300


def test_ties_of_the_rebase_test_are_decided(nm):
    """A 1280x720 part of the 1920x1080x16 view at 1e-12: past a near return of the
    orbit to 0 a whole region's |Y| and |delta| agree to 2^-19.  Without the jumps
    6.3 % of the samples need the FP64 kernel."""
    view = dict(C2, nr=720, nc=1280, sc=1, step="1.302083333333333e-16")
    m = setup_gpu(nm, view, path=nm.PATH_FE32, keep64=False)
    m.precompute()
    m.render()
    share = m.stat(nm.STAT_FP64_REWORK) / (720 * 1280)
    print("rework %.4f" % share)
    assert share <= 1.05 * 0.0631


# (view, the largest difference of the path without jumps)
DEEP = ("-0.743643887037229095312187703165620156203167189531343718751406",
        "0.131825904205267520317187749964062031515607811562296900001563")


@pytest.mark.parametrize("view,bar", [
    (dict(nr=1200, nc=1600, cre=C2["cre"], cim=C2["cim"], step="1.25e-16", N=20000), 4.82e-5),
    (dict(nr=1080, nc=1920, cre=DEEP[0], cim=DEEP[1], step="5.208333333333333e-24", N=50000,
          center=True), 2.83e-5),
], ids=["2e-13", "1e-20"])
def test_smoothing_is_as_near_as_without_jumps(nm, view, bar):
    out = []
    for path in (nm.PATH_FP64, nm.PATH_FE32):
        m = setup_gpu(nm, dict(view, sc=1, tol=1e-10), path=path)
        if view.get("center"):
            m.set_option(nm.OPT_REFERENCE, nm.REFERENCE_CENTER)
        m.precompute()
        m.render()
        out.append((m.grid()["iterations"].copy(), m.smoothing64().copy()))
    (i0, s0), (i1, s1) = out
    assert np.array_equal(i0, i1)
    d = np.abs(s0 - s1).max()
    print("largest difference %.3g" % d)
    assert d <= bar


def test_tables_are_found_after_a_change_of_path(nm):
    """A view precomputed and uploaded for the FP64 path, which reads no jumps, gets
    them when it first renders on the FE32 path: the steps and the grid of a view that
    was precomputed for it."""
    view = dict(nr=400, nc=600, sc=1, cre=DEEP[0], cim=DEEP[1], step="2e-23", N=20000, tol=1e-10)
    got = []
    for first in (nm.PATH_FE32, nm.PATH_FP64):
        m = setup_gpu(nm, view, path=first, keep64=False)
        m.set_option(nm.OPT_REFERENCE, nm.REFERENCE_CENTER)
        m.precompute()
        if first == nm.PATH_FP64:
            m.render()
            fp64 = m.grid()["iterations"].copy()
            steps64 = m.stat(nm.STAT_EXECUTED_ITERS)
            m.set_path(nm.PATH_FE32)
        m.render()
        got.append((m.grid().copy(), m.stat(nm.STAT_EXECUTED_ITERS)))
    assert np.array_equal(got[0][0], got[1][0]) and got[0][1] == got[1][1]
    assert np.array_equal(fp64, got[0][0]["iterations"])
    assert got[0][1] < 0.8 * steps64  # steps were jumped
