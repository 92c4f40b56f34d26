"""CPU checks of the 3-D kernels' carried walks through their host model
(tests/native/dd_walk3d.cpp): rows and slices merged in ascending z, 2 to 8 rows
and 8 or 16 slices a thread.  The bar of the other host model: rel-L2 <= 1e-6
against the FP32 oracle, and the pairs exact transposes of each other.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import cases3d
from conftest import _G3, ROOT, rel_l2

CASES = cases3d.cases()
OPS = {"proj": 0, "proj_t": 1, "bproj": 2, "bproj_t": 3, "bproj_w": 4, "bproj_tw": 5}
SCAN = {"cone_flat": 0, "cone_arc": 1, "spiral": 2}


@pytest.fixture(scope="module")
def walk():
    src = os.path.join(ROOT, "tests", "native", "dd_walk3d.cpp")
    so = os.path.join(ROOT, "tests", "native", "_build", "libddwalk3d.so")
    os.makedirs(os.path.dirname(so), exist_ok=True)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", src, "-o", so], check=True)
    lib = ctypes.CDLL(so)
    fp = ctypes.POINTER(ctypes.c_float)
    lib.walk_apply3d.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.POINTER(_G3), fp, fp, fp, fp] + [ctypes.c_int] * 4

    def apply(case, op, x, rows, slices):
        geom, opt, ang, sp = case
        o = [float(v) for v in opt]
        if geom == "spiral":
            o = o[:14] + [0.0] + o[14:]
        g = _G3(*[int(v) for v in o[:5]], *o[5:])
        V, B = len(ang), x.shape[0]
        shape = (B, V, g.num_row, g.num_col) if op in cases3d.IMAGE_IN else (B, g.depth, g.height, g.width)
        out = np.zeros(shape, np.float32)
        ptr = lambda a: None if a is None else np.ascontiguousarray(a, np.float32).ctypes.data_as(fp)   # noqa: E731
        arrays = [np.ascontiguousarray(a, np.float32) if a is not None else None for a in (ang, sp, x)]
        assert lib.walk_apply3d(SCAN[geom], OPS[op], ctypes.byref(g), *[ptr(a) for a in arrays], out.ctypes.data_as(fp), B, V,
                                rows, slices) == 0
        return out
    return apply


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("op", cases3d.OPS)
def test_walk_matches_oracle(walk, oracle_mod, name, op):
    geom, opt, ang, sp = CASES[name]
    x, y = cases3d.inputs(CASES[name], batch=1, seed=3)
    inp = x if op in cases3d.IMAGE_IN else y
    ref = oracle_mod.run3d(geom, op, inp, ang, opt, source_pos=sp, prec="f", nthreads=4)
    for rows, slices in ((8, 16), (2, 8)):
        assert rel_l2(walk(CASES[name], op, inp, rows, slices), ref) <= 1e-6


@pytest.mark.parametrize("name", ["cone_flat_small", "spiral_small"])
def test_walk_pairs_are_exact_transposes(walk, name):
    x, y = cases3d.inputs(CASES[name], batch=1, seed=5)
    for fwd, adj in (("proj", "proj_t"), ("bproj_t", "bproj"), ("bproj_tw", "bproj_w")):
        ax = walk(CASES[name], fwd, x, 4, 16).astype(np.float64)
        aty = walk(CASES[name], adj, y, 4, 16).astype(np.float64)
        lhs, rhs = float((ax * y).sum()), float((x * aty).sum())
        assert abs(lhs - rhs) <= 1e-6 * abs(lhs)
