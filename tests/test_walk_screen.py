"""The device walk's FP32 opening test must repeat every test in FP64 whose
squared distance lies within its error of the threshold.  The split centres
(FP32 and BF16 parts), the FP32 distances and the margin of csrc/walk.cu are
restated here with its constants, and the margin is held against the FP64
distances of the host walk over random centres and boxes, also where the
margin is smallest against the error: structure of 2^-24 to 2^-10 of its
distance from the origin."""
import os
import re

import numpy as np
import pytest

F = np.float32
SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "changa_gb300",
                   "csrc", "walk.cu")


def constants():
    names = {"kU": 2.0 ** -24}
    with open(SRC) as f:
        for k, v in re.findall(r"constexpr (?:float|double) (kScreen\w*) = ([^;]+);", f.read()):
            names[k] = eval(re.sub(r"(?<=[\d.])f\b", "", v), {}, dict(names))
    return names


def bf16(x, up=False):
    b = np.asarray(x, F).view(np.uint32).astype(np.uint64)
    b = b + 0xffff if up else b + 0x7fff + ((b >> 16) & 1)
    return (b & 0xffff0000).astype(np.uint32).view(F)


def split(x):
    hi = x.astype(F)
    return hi, bf16((x - hi).astype(F))


def distances(c, lo, hi, o, k):
    """FP32 near and far squared distances and E; the FP64 ones."""
    m, h = 0.5 * (lo + hi), 0.5 * (hi - lo)
    mx, hx = np.abs(m).max(1), np.abs(h).max(1)
    eps = k["kScreenH"] * hx + k["kScreenM"] * (mx + hx)
    E = bf16((k["kScreenE"] * eps * eps + 1e-37).astype(F), up=True)
    eo = 4.0 * k["kU"] * np.abs(o).max()
    E = E + F(1.001 * k["kScreenE"] * eo * eo)
    (ch, cl), (mh, ml) = split(c), split(m)
    d = np.abs((ch - mh) + o.astype(F) + (cl - ml))
    hf = h.astype(F)
    near = np.maximum(F(0), d - hf)
    far = d + hf
    x = c + o
    near64 = np.maximum(0.0, np.maximum(lo - x, x - hi))
    far64 = np.maximum(np.abs(x - lo), np.abs(hi - x))
    return [((a * a).sum(1, dtype=F), (b * b).sum(1), E) for a, b in
            ((near, near64), (far, far64))]


@pytest.mark.parametrize("at", [0.0, 1.0, 520.0, -1e6])
@pytest.mark.parametrize("period", [0.0, 0.7])
def test_margin_covers_the_error(at, period):
    k = constants()
    assert {"kScreen", "kScreenE", "kScreenH", "kScreenM"} <= set(k)
    rng = np.random.default_rng(7)
    for log in range(-24, -9) if at else (-10, 0, 10):
        ext = (abs(at) or 1.0) * 2.0 ** log
        n = 20000
        c = at * rng.uniform(0.5, 1.0, 3) + ext * rng.uniform(-1, 1, (n, 3))
        mid = at * rng.uniform(0.9, 1.0) + ext * rng.uniform(-1, 1, (n, 3))
        mid = np.where(rng.random((n, 1)) < 0.5, mid, c + ext * rng.normal(0, 0.3, (n, 3)))
        half = ext * 2.0 ** rng.uniform(-12, 0, (n, 1)) * rng.uniform(0.1, 1, (n, 3))
        o = period * abs(at or 1.0) * rng.integers(-1, 2, (n, 3)).astype(np.float64)
        c = np.where(rng.random((n, 1)) < 0.7, c - o, c)  # near across the boundary too
        for v, v64, E in distances(c, mid - half, mid + half, o, k):
            # both sides of screen_le leave at least |v - v64| to the threshold
            room = k["kScreen"] * v.astype(np.float64) + E
            assert (np.abs(v - v64) <= room).all(), (log, (np.abs(v - v64) / room).max())
