"""Calls at the limits of what the entry points accept, on the GPU.

Bars as for the same operators elsewhere: rel-L2 <= 1e-5 against the FP32
oracle in 2-D, 5e-5 in 3-D.
"""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from test_gpu_2d import run as run2d

pytestmark = pytest.mark.gpu


# The source inside the image's rectangle: a line level with it or behind it
# meets nothing (its boundaries would descend), the lines before it are what
# they are without the others.
@pytest.mark.parametrize("view", [0.1, 0.7, 1.5, 2.4, 3.2, 4.0, 4.8, 5.6])
@pytest.mark.parametrize("geom,op,B", [("flat", "proj", 1), ("flat", "bproj_t", 8), ("arc", "proj", 2), ("arc", "bproj_tw", 3)])
def test_source_inside_the_image(oracle_mod, geom, op, B, view):
    W, H, D, sid = 300, 260, 90, 100.0
    opt = [W, H, D, 1.0, 0.9, 1.0 * (2.0 if geom == "flat" else 1.0 / sid), sid, 2 * sid, 0.0, 0.0, 0.0]
    ang = np.array([view], np.float32)
    rng = np.random.default_rng(int(10 * view))
    x = rng.random((B, H, W), dtype=np.float32)
    # the source stands at (-sin, cos) sid; rows are walked where cos^2 > 1/2
    rows, cols = (H / 2 - np.arange(H) - 0.5) * 0.9, np.arange(W) - W / 2 + 0.5
    sx, sy = -np.sin(view) * sid, np.cos(view) * sid
    if np.cos(view) ** 2 > 0.5:
        front = np.broadcast_to(((rows < sy) if sy > 0 else (rows > sy))[:, None], (H, W))
    else:
        front = np.broadcast_to(((cols < sx) if sx > 0 else (cols > sx))[None], (H, W))
    assert not front.all()
    ref = oracle_mod.run2d(geom, op, x * front, ang, opt, nthreads=8)
    out = run2d(geom, op, x, ang, opt)
    assert np.any(ref) and rel_l2(out, ref) <= 1e-5
    assert np.array_equal(run2d(geom, op, x * front, ang, opt), out)
    # and the transpose puts nothing behind it
    adj = {"proj": "proj_t", "bproj_t": "bproj", "bproj_tw": "bproj_w"}[op]
    y = rng.standard_normal((B, 1, D)).astype(np.float32)
    b = run2d(geom, adj, y, ang, opt)
    assert not b[:, ~front].any()
    lhs, rhs = float((out.astype(np.float64) * y).sum()), float((x * b.astype(np.float64)).sum())
    # each side's FP32 sums: some 30 roundings of 2^-24 of the magnitudes, on either
    assert abs(lhs - rhs) <= 5e-6 * float(np.abs(out.astype(np.float64) * y).sum())
