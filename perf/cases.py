"""The work that the speed of this framework is measured on.

Each case is one call, or one short run of calls, that a program using the
framework makes over and over: rendering a row, a window, a still image or the
frames of a zoom, at the zoom depths, grid sizes, iteration counts and paths
that are used in earnest.  Escape counts depend on the view alone, so a case's
inputs are its view; a seed moves the center by at most 2 % of the width.

Sizes come from the repository's tests and benchmark (the 640x480 view of
width 3, the 1920x1080 view with 4x4 samples at width 1e-12, the 3840x2160 view
at width 1e-300, the 1280x720 zoom video) or are common window and image sizes.
"""
import os
import random
import tempfile
from decimal import Decimal, getcontext
from fractions import Fraction

import numpy as np
import torch

import newman_gb300 as nm

# The center of the 1e-12 view (and of the zoom video above the double range).
SEAHORSE = ("-0.743643887037151", "0.131825904205330")
# The center of the 1e-300 view: a point on the boundary at every width above it.
DEEP_RE = ("-0.743643887037229095312187703165620156203167189531343718751406171826566093812504689"
           "062796887503281078085934374921925001718624951561718906221874687046864066405921878121"
           "562828123436718265675001249562460933125031242186875171831250780874981247812390626560"
           "624843796873906531285942343468732814531093798432968421875")
DEEP_IM = ("0.1318259042052675203171877499640620315156078115622969000015629687765646874531156210"
           "934843421850004844203078128750015624998281593775003437171917188280749959375312468699"
           "996718796875001875234409378593781296878749640635934218609398434218703110937812687503"
           "12062495316250046887502499515615625312187496879062000000")

PATHS = {"reference": nm.PATH_REFERENCE, "fp64": nm.PATH_FP64, "fe32": nm.PATH_FE32,
         "mp": nm.PATH_MP}

# A palette in the reference's text format (two hue cycles, a saturation cycle,
# two luminance waves).
PALETTE = """2
3 10.0 130.5 250.25 90
2 300.0 45.0 60
70

3
0.9 0.4 0.7
33

2
1.5 40
0.75 13
"""


def listed():
    return [
        # the smallest call: one row of a window, as the reference's viewer
        # renders and shows a view row by row
        dict(name="row_640", kind="row", rows=480, cols=640, width="3.0", N=1024, row=150),
        # an interactive window at the start of a zoom: the reference's double loop
        dict(name="window_640x480", kind="frame", path="reference", center="whole", rows=480,
             cols=640, sc=1, width="3.0", N=1024),
        # a still image of a shallow zoom, multisampled and coloured, odd sizes
        dict(name="still_1367x769_2x2", kind="still", path="reference", center="seahorse",
             rows=769, cols=1367, sc=2, width="3e-5", N=5000),
        # a double-loop view near the end of the double range: the last steps of
        # a zoom before perturbation takes over
        dict(name="double_800x600_1e-9", kind="frame", path="reference", center="seahorse",
             rows=600, cols=800, sc=1, width="1e-9", N=10000),
        # a small odd window of a deep zoom, while the user looks for a view
        dict(name="window_333x517_1e-20", kind="frame", path="fe32", center="deep", rows=333,
             cols=517, sc=1, width="1e-20", N=20000),
        # a multisampled still image just below the double range: the benchmark's
        # main view
        dict(name="still_1080p_4x4_1e-12", kind="frame", path="fe32", center="seahorse",
             rows=1080, cols=1920, sc=4, width="1e-12", N=50000),
        # a 4K image beyond the double exponent range
        dict(name="still_4k_1e-300", kind="frame", path="fe32", center="deep", rows=2160,
             cols=3840, sc=1, width="1e-300", N=1000000),
        # the same kind of image in plain FP64 perturbation
        dict(name="fp64_961x541_1e-12", kind="frame", path="fp64", center="seahorse", rows=541,
             cols=961, sc=2, width="1e-12", N=50000),
        # the reference's own arbitrary-precision results at its smallest precision
        dict(name="exact_960x540_1e-12", kind="frame", path="mp", center="seahorse", rows=540,
             cols=960, sc=2, width="1e-12", N=50000),
        # and deeper, where values take more limbs
        dict(name="exact_401x301_1e-38", kind="frame", path="mp", center="deep", rows=301,
             cols=401, sc=1, width="1e-38", N=100000),
        # one step of a deep zoom: a new view, its reference orbit, the render and
        # the multisampled frame on the host
        dict(name="zoom_step_800x600_2x2", kind="step", path="fe32", center="seahorse", rows=600,
             cols=800, sc=2, width="2e-13", N=20000),
        # a zoom video: every frame's own view in one launch sequence
        dict(name="video_24x640x360_2x2", kind="video", frames=24, rows=360, cols=640, sc=2,
             width="4.0", width_end="1e-40", N=1000, N_end=100000),
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi], odd ones among them."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _width(rng, lo, hi):
    """A width 10^-e, e uniform in [lo, hi]."""
    e = rng.uniform(lo, hi)
    n = int(e // 1)
    return "%.4fe-%d" % (10 ** (n + 1 - e), n + 1) if e >= 0 else "%.4f" % 10 ** -e


def draw(rng):
    kind = rng.choice(["row", "frame", "still", "deep", "deep", "fp64", "exact", "step", "video"])
    rows, cols = _log(rng, 48, 1100), _log(rng, 64, 1940)
    if kind == "row":
        return dict(kind="row", center="seahorse", rows=rows, cols=cols, width=_width(rng, -0.5, 4), row=rows // 2,
                    N=_log(rng, 256, 8192))
    if kind in ("frame", "still"):
        return dict(kind=kind, path="reference", center="seahorse", rows=rows, cols=cols,
                    sc=rng.choice([1, 1, 2, 3]), width=_width(rng, -0.5, 9), N=_log(rng, 500, 10000))
    if kind == "step":
        return dict(kind="step", path="fe32", center="seahorse", rows=_log(rng, 48, 600),
                    cols=_log(rng, 64, 800), sc=rng.choice([1, 2, 3]), width=_width(rng, 13.7, 15),
                    N=_log(rng, 10000, 50000))
    if kind == "video":
        return dict(kind="video", frames=rng.randint(3, 16), rows=_log(rng, 64, 360),
                    cols=_log(rng, 96, 640), sc=rng.choice([1, 2]), width="4.0",
                    width_end=_width(rng, 12, 60), N=1000, N_end=_log(rng, 20000, 150000))
    # the reference renders samples down to a step of 1e-45
    e = rng.uniform(14.5, 40 if kind == "exact" else 60)
    width = "%.4fe-%d" % (10 ** (int(e) + 1 - e), int(e) + 1)
    N = _log(rng, 20000 + 1500 * int(e - 14), 200000)
    if kind == "deep":
        return dict(kind="frame", path="fe32", center="deep", rows=rows, cols=cols,
                    sc=rng.choice([1, 1, 2]), width=width, N=N)
    return dict(kind="frame", path="fp64" if kind == "fp64" else "mp", center="deep",
                rows=_log(rng, 48, 541), cols=_log(rng, 64, 961), sc=1, width=width, N=N)


# ---- preparation ---------------------------------------------------------------

def _center(case, seed):
    """The case's center, moved by up to 2 % of the width."""
    getcontext().prec = 400
    name = case.get("center", "whole")
    re, im = {"whole": ("-0.75", "0"), "seahorse": SEAHORSE, "deep": (DEEP_RE, DEEP_IM)}[name]
    rng = random.Random(seed)
    w = Decimal(case.get("width_end", case["width"]))
    return [str(Decimal(v) + w * Decimal(rng.randint(-10**9, 10**9)) * Decimal("2e-11"))
            for v in (re, im)]


def _step(width, cols):
    getcontext().prec = 40
    return str(Decimal(width) / cols)


def _view(case, center, width, N, path):
    sc = case.get("sc", 1)
    m = nm.Mandelbrot(case["rows"] * sc, case["cols"] * sc)
    step = _step(width, case["cols"] * sc)
    m.set_view(center[0], center[1], step, step, N)
    m.set_path(PATHS[path])
    # a reference orbit at the view center where the search for a longer one
    # would take longer than the render
    if Decimal(width) < Decimal("1e-16"):
        m.set_option(nm.OPT_REFERENCE, nm.REFERENCE_CENTER)
    return m


class _DeviceGrid:
    """The escape grid on the GPU ({int32, float32} per sample) as the framework holds it."""

    def __init__(self, m):
        p, _ = m.device_grid()
        self.owner = m
        self.__cuda_array_interface__ = {"shape": (m.rows(), m.cols(), 2), "typestr": "<i4",
                                         "data": (p, False), "version": 3}


def _grid(m):
    g = torch.as_tensor(_DeviceGrid(m), device="cuda")
    return {"iterations": g[..., 0], "smoothing": g[..., 1].view(torch.float32)}


def prepare(case, seed):
    nm.load_library()
    torch.cuda.init()
    kind, center = case["kind"], _center(case, seed)
    s = {"case": case}
    if kind == "video":
        getcontext().prec = 60
        s["batch"] = nm.Batch(sc=case["sc"])
        w0, w1 = Decimal(case["width"]), Decimal(case["width_end"])
        for k in range(case["frames"]):
            t = Decimal(k) / (case["frames"] - 1)
            getcontext().prec = 60
            w = w0 * (w1 / w0) ** t
            N = int(round(case["N"] + (case["N_end"] - case["N"]) * float(t)))
            m = _view(case, center, str(w), N, "fe32")
            if m.useHardware():
                m.set_path(nm.PATH_REFERENCE)
            else:
                m.set_option(nm.OPT_REFERENCE, nm.REFERENCE_CENTER)
                m.precompute()
            s["batch"].add(m)
        return s
    path = case.get("path", "reference")
    m = s["view"] = _view(case, center, case["width"], case["N"], path)
    if kind == "step":
        s["center"], s["step"] = center, _step(case["width"], case["cols"] * case["sc"])
        s["out"] = np.empty((case["rows"], case["cols"]), nm.ESCAPE_DTYPE)
    elif path != "reference":
        m.precompute()
        m.upload()
    if kind == "still":
        fd, name = tempfile.mkstemp(suffix=".pal")
        with os.fdopen(fd, "w") as f:
            f.write(PALETTE)
        s["palette"] = nm.Palette(name)
        os.unlink(name)
    return s


def _mean_value(frame):
    """The mean escape value of each pixel, which a reduced frame holds as its
    whole part and the rest (one float, split)."""
    return frame["iterations"].astype(np.float32) + frame["smoothing"]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "video":
        state["batch"].render()
        return [_mean_value(f) for f in state["batch"].frames_out()]
    m = state["view"]
    if kind == "row":
        m.computeRow(case["row"])
        return _grid(m)
    if kind == "step":
        m.set_view(state["center"][0], state["center"][1], state["step"], state["step"], case["N"])
        m.precompute()
        m.render()
        return {"frame": _mean_value(m.reduce(case["sc"], state["out"])), "samples": _grid(m)}
    m.render()
    out = _grid(m)
    if kind == "still":
        out["image"] = m.colorize(state["palette"], sc=case["sc"], smooth=True)
    return out


def work(case):
    """Every sample's escape value is written once (8 bytes; a pixel's 8 or 3
    bytes more where the case makes an image of them) and takes at least one
    step Z = Z^2 + C (3 products, 4 sums).  The steps a sample really takes
    depend on the view, not on the case's numbers."""
    pixels = case["cols"] * (1 if case["kind"] == "row" else case["rows"])
    n = pixels * case.get("sc", 1) ** 2 * case.get("frames", 1)
    extra = {"still": 3, "step": 8, "video": 8}.get(case["kind"], 0) * pixels * case.get("frames", 1)
    return {"bytes": 8 * n + extra, "flops": 7 * n}


# ---- 64-bit values -------------------------------------------------------------

def _trunc(x):
    """A Fraction truncated toward zero to a double."""
    d = float(x)
    if abs(Fraction(d)) > abs(x):
        d = float(np.nextafter(d, 0.0))
    return d


def exact(case, seed):
    """Smoothing values of the double-loop views, from a plain elementwise loop
    in 64 bits.  Views below the double range have none: what their samples
    give depends on more than 64 bits of the coordinates."""
    if case["kind"] not in ("row", "frame", "still") or case.get("path", "reference") != "reference":
        return None
    sc = case.get("sc", 1)
    nr, nc, N = case["rows"] * sc, case["cols"] * sc, case["N"]
    # chaotic at the scale of a double's rounding: the last bit of a coordinate decides
    if Decimal(case["width"]) / nc < Decimal("1e-9") or nr * nc > 5_000_000:
        return None
    center = [Fraction(Decimal(v)) for v in _center(case, seed)]
    step = Fraction(Decimal(_step(case["width"], nc)))
    cre = torch.tensor([_trunc(center[0] + (c - nc // 2) * step) for c in range(nc)],
                       dtype=torch.float64, device="cuda")
    rows = [case["row"]] if case["kind"] == "row" else range(nr)
    cim = torch.tensor([_trunc(center[1] + (nr // 2 - r - 1) * step) for r in rows],
                       dtype=torch.float64, device="cuda")
    x0 = cre[None, :].expand(len(cim), nc).reshape(-1)
    y0 = cim[:, None].expand(len(cim), nc).reshape(-1)
    smooth = torch.zeros(x0.numel(), dtype=torch.float64, device="cuda")
    q = (x0 - 0.25) ** 2 + y0 * y0
    inside = (q * (q + x0 - 0.25) < 0.25 * y0 * y0) | ((x0 + 1) ** 2 + y0 * y0 < 0.0625)
    at = torch.nonzero(~inside).reshape(-1)
    x0, y0 = x0[at], y0[at]
    x, y = x0, y0
    for i in range(N):
        x, y = (x * x - y * y) + x0, (x + x) * y + y0
        r2 = x * x + y * y
        out = r2 > 1048576.0
        if bool(out.any()):
            smooth[at[out]] = 1.0 - torch.log2(0.5 * torch.log(r2[out]) / np.log(1024.0))
            keep = ~out
            at, x0, y0, x, y = at[keep], x0[keep], y0[keep], x[keep], y[keep]
            if not at.numel():
                break
    grid = torch.zeros(nr, nc, dtype=torch.float64, device="cuda")
    if case["kind"] == "row":
        grid[case["row"]] = smooth
    else:
        grid = smooth.reshape(nr, nc)
    got = {"iterations": None, "smoothing": grid}
    if case["kind"] == "still":
        got["image"] = None
    return got
