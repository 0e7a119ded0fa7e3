"""The FE32 path's exponent renormalisation interval (NM_OPT_RENORM) counts a
sample's own steps: the pass pipeline, whose warps advance their samples in pieces
that depend on one another, gives the bits of the single-pass kernel and of any
number of blocks."""
import json
import os
from decimal import Decimal

import numpy as np
import pytest

from helpers import setup_gpu, step_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nm():
    import newman_gb300
    newman_gb300.load_library()
    return newman_gb300


def test_renormalisation_follows_the_sample(nm):
    steps = json.load(open(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden",
                                        "deep_centers.json")))["steps"]
    at = steps[next(i for i, s in enumerate(steps) if Decimal(s["width"]) <= Decimal("1e-330")) - 1]
    view = dict(nr=96, nc=160, sc=2, cre=at["next_center_re"], cim=at["next_center_im"],
                step=step_for("1e-330", 160), N=300000, tol=1e-10)
    m = setup_gpu(nm, view, path=nm.PATH_FE32, keep64=False)
    m.set_option(nm.OPT_REFERENCE, nm.REFERENCE_CENTER)
    m.precompute()
    # around the pieces of 16 steps: below, not a multiple, the default, the largest
    for renorm in (5, 24, 0, 256):
        grids, rework = [], []
        for single, blocks in ((1, 0), (0, 0), (0, 3)):
            m.set_option(nm.OPT_RENORM, renorm)
            m.set_option(nm.OPT_FE32_SINGLE_PASS, single)
            m.set_option(nm.OPT_BLOCKS, blocks)
            m.render()
            grids.append(m.grid().copy())
            rework.append(m.stat(nm.STAT_FP64_REWORK))
        assert rework[0] == rework[1] == rework[2] and 0 < rework[0] < grids[0].size, renorm
        for g in grids[1:]:
            assert np.array_equal(g, grids[0]), renorm
