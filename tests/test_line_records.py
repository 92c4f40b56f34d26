"""CPU check of the 2-D walked-line records and of the boundary tables that the
forward's producer warps build from them (tests/native/dd_records.cpp): every
run of boundaries lies inside its line, every write inside its table, and the
tables hold the drifted sequence.  Lines level with the source or behind it
(a source inside the image's rectangle) and boundaries that a pitch below half
an ulp leaves standing must give records that can be walked like any other.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, _G2


@pytest.fixture(scope="module")
def records():
    src = os.path.join(ROOT, "tests", "native", "dd_records.cpp")
    so = os.path.join(ROOT, "tests", "native", "_build", "libddrecords.so")
    os.makedirs(os.path.dirname(so), exist_ok=True)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", src, "-o", so], check=True)
    lib = ctypes.CDLL(so)
    fp, lp = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_longlong)
    lib.records_check.argtypes = [ctypes.c_int, ctypes.POINTER(_G2), fp, ctypes.c_int, lp]

    def check(geom, W, H, D, pix, cell, sid, shift=0.0, views=40):
        det = cell * {0: 1.0, 1: 1085.6 / 595.0, 2: 1.0 / sid}[geom]
        g = _G2(W, H, D, pix, 0.9 * pix, det, sid, sid * 1085.6 / 595.0, shift, -shift, 0.1 * det)
        ang = (np.arange(views) * 2 * np.pi / views + 0.05).astype(np.float32)
        out = (ctypes.c_longlong * 6)()
        assert lib.records_check(geom, ctypes.byref(g), ang.ctypes.data_as(fp), views, out) == 0
        return dict(zip(("lines", "ascending", "bad_runs", "bad_writes", "kept", "ulps"), out))
    return check


@pytest.mark.parametrize("geom", [0, 1, 2])
@pytest.mark.parametrize("W,H,D,pix,cell,sid,shift", [
    (67, 93, 150, 0.7, 1.0, 595.0, 0.3),
    (1, 1, 1, 1.0, 1.0, 595.0, 0.0),
    (4096, 3, 40, 0.2, 20.0, 595.0, 0.0),
    (300, 260, 200, 1.0, 1.5, 100.0, 0.0),      # the source inside the image
    (64, 64, 90, 2.0, 2.0, 31.0, 0.0),          # ... level with a line at some views
    (300, 260, 200, 1.0, 1.5, 0.01, 0.0),       # ... at its centre
    (64, 48, 90, 1e-3, 1e-3, 595.0, 4e4),       # a pitch below half an ulp: boundaries stand still
])
def test_records_stay_inside_their_lines(records, geom, W, H, D, pix, cell, sid, shift):
    r = records(geom, W, H, D, pix, cell, sid, shift)
    assert r["bad_runs"] == 0 and r["bad_writes"] == 0 and r["kept"] == 0
    assert r["ascending"] == r["lines"] or (geom and sid < 200.0) or shift > 1e3
    # a table's run of equal steps settles a round-to-even tie after one step
    assert r["ulps"] <= 1
