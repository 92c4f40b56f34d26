"""The kernels at the edges of their splits, against the FP32 oracle.

2-D forward: groups of 8, 4, 2 and 1 slices and their remainders, the prefix
sums of one and two, every class of detector passes, lines too long for 8
slices.  2-D adjoints: clusters whose CTAs get no view, views of one axis
only, partial tiles, lines shorter than a warp.  3-D forward: 2, 4 and 8 rows
a thread with a remainder of rows, windows of more than one chunk of slices,
cells of many pixels.  3-D adjoint: 8 and 16 slices a thread, volumes in a
pair and alone.

Bars as for the same operators elsewhere: rel-L2 <= 1e-5 in 2-D, where the
oracle is bit-exact with the reference's CPU code; <= 5e-5 in 3-D, where the
oracle rounds its trigonometry differently from device code.
"""
import numpy as np
import pytest
import torch

from cases3d import IMAGE_IN, spiral_source
from conftest import rel_l2
from test_gpu_2d import run as run2d
from test_gpu_3d import run as run3d

pytestmark = pytest.mark.gpu


def _check2d(oracle_mod, geom, op, W, H, D, ang, B, cell=1.4, seed=0):
    """cell: a detector cell at the isocentre, in pixels."""
    pix = 0.7
    det = cell * pix * {"para": 1.0, "flat": 1085.6 / 595.0, "arc": 1.0 / 595.0}[geom]
    opt = [W, H, D, pix, 0.9 * pix, det, 595.0, 1085.6, 0.1, -0.2, 0.1 * det]
    ang = np.asarray(ang, np.float32)
    rng = np.random.default_rng(seed)
    x = rng.random((B, H, W), dtype=np.float32) if op in IMAGE_IN else \
        rng.standard_normal((B, ang.size, D)).astype(np.float32)
    ref = oracle_mod.run2d(geom, op, x, ang, opt, nthreads=8)
    assert np.any(ref)
    assert rel_l2(run2d(geom, op, x, ang, opt), ref) <= 1e-5


def _turn(V):
    return np.arange(V) * 2 * np.pi / V + 0.1


@pytest.mark.parametrize("B", [1, 2, 3, 4, 5, 8, 9, 15])
@pytest.mark.parametrize("geom,op", [("para", "proj"), ("flat", "proj"), ("flat", "bproj_t"), ("arc", "bproj_tw")])
def test_forward_slice_groups(oracle_mod, geom, op, B):
    _check2d(oracle_mod, geom, op, 67, 93, 150, _turn(9), B, seed=B)


# 248 bins a pass: the last bin of a pass, the first of the next; cells of
# many pixels and many cells a pixel; lines too long for 8 slices
@pytest.mark.parametrize("W,H,D,cell", [(40, 31, 248, 0.3), (40, 31, 249, 0.3), (40, 64, 497, 0.2), (33, 64, 745, 0.1),
                                        (33, 40, 993, 0.08), (150, 97, 12, 17.0), (1300, 5, 300, 5.0), (1, 9, 40, 1.0)])
@pytest.mark.parametrize("geom,B", [("para", 1), ("flat", 2), ("arc", 3), ("flat", 8)])
def test_forward_detector_passes_and_lines(oracle_mod, geom, B, W, H, D, cell):
    if geom != "para" and W > 1000:
        W = 1100   # inside the source circle
    _check2d(oracle_mod, geom, "proj", W, H, D, _turn(5), B, cell, seed=D)


# a cluster's 4 CTAs share the views: fewer views than CTAs, one axis only
@pytest.mark.parametrize("angles", [[0.05], [1.5], [0.1, 1.6, 3.0], [0.0, 0.2, -0.3, 3.1, 0.4, 0.1, -0.2], list(_turn(37))],
                         ids=["one_x", "one_y", "three", "one_axis", "turn"])
@pytest.mark.parametrize("geom,op", [("para", "proj_t"), ("para", "bproj"), ("flat", "proj_t"), ("arc", "bproj_w")])
@pytest.mark.parametrize("W,H,B", [(33, 65, 1), (64, 32, 4), (31, 97, 5), (3, 40, 2)])
def test_adjoint_clusters(oracle_mod, geom, op, angles, W, H, B):
    _check2d(oracle_mod, geom, op, W, H, 90, angles, B, seed=W)


@pytest.mark.parametrize("scan", ["flat", "para"])
def test_uneven_batch_of_many_slices(scan):
    """1 to 9 slices an instance: items of 1, 2 and 4 slices, line items."""
    import pridediff_gb300 as P
    from pridediff_gb300.batch import UnevenBatch2d
    sizes, batch = [(64, 48), (33, 70), (96, 96), (40, 40)], [1, 3, 9, 4]
    projs = [P.projector2d(s, 100 + 10 * i, 0.66, 1.2858, 595.0, 1085.6, scan_type=scan).cuda()
             for i, s in enumerate(sizes)]
    angs = [torch.arange(v, dtype=torch.float32, device="cuda") * (2 * np.pi / v) for v in (3, 20, 45, 1)]
    ub = UnevenBatch2d(projs, angs, batch)
    g = torch.Generator(device="cuda").manual_seed(5)
    xs = [torch.rand(s, device="cuda", generator=g) for s in ub.img_shapes]
    rs = [torch.randn(s, device="cuda", generator=g) for s in ub.sino_shapes]
    ys, bs = ub.unpack_sinos(ub.forward(ub.pack(xs))), ub.unpack_images(ub.adjoint(ub.pack(rs)))
    for p, a, x, y, r, b in zip(projs, angs, xs, ys, rs, bs):
        # the two forwards' roundings, each within 1e-5 of exact arithmetic
        assert rel_l2(y.cpu().numpy(), p.projection(x, a).cpu().numpy()) <= 2e-5
        assert torch.equal(b, p.projection_t(r, a))


def _check3d(oracle_mod, geom, op, W, H, dep, cols, rows, V, B, cell=1.5, pz=1.0, row=1.5, sid=300.0):
    col = cell * 2 * (1.0 if geom == "cone_flat" else 0.5 / sid)
    opt = [W, H, dep, cols, rows, 1.0, 1.1, pz, col, row, sid, 2 * sid, 0.3, -0.2]
    opt += [0.1 * col, 0.3] if geom == "spiral" else [0.4, 0.1 * col, 0.3]
    opt = np.array(opt, np.float32)
    ang = _turn(V).astype(np.float32)
    sp = spiral_source(V, 0.5, -0.25 * V) if geom == "spiral" else None
    rng = np.random.default_rng(rows + B)
    x = (rng.random((B, dep, H, W)) if op in IMAGE_IN else rng.random((B, V, rows, cols))).astype(np.float32)
    ref = oracle_mod.run3d(geom, op, x, ang, opt, source_pos=sp, nthreads=8)
    assert np.any(ref)
    assert rel_l2(run3d(geom, op, x, ang, opt, sp), ref) <= 5e-5


@pytest.mark.parametrize("rows", [1, 16, 17, 33, 64, 65, 129])
@pytest.mark.parametrize("geom,op,B", [("cone_flat", "proj", 1), ("cone_arc", "bproj_t", 2), ("spiral", "proj", 3)])
def test_forward3d_rows(oracle_mod, geom, op, B, rows):
    _check3d(oracle_mod, geom, op, 37, 44, 20, 45, rows, 5, B, row=60.0 / rows)


# thin slices (a cell row's window spans chunks), cells of 12 pixels, cells
# far below a pixel, two walk blocks, more than a tile's pixels in 32 columns
@pytest.mark.parametrize("W,H,dep,cols,cell,pz", [(40, 33, 300, 30, 1.5, 0.1), (150, 97, 9, 14, 12.0, 1.0),
                                                  (40, 40, 9, 300, 0.2, 1.0), (130, 130, 5, 70, 3.0, 1.0),
                                                  (1, 40, 3, 40, 1.5, 1.0)])
@pytest.mark.parametrize("geom,op,B", [("cone_flat", "proj", 2), ("spiral", "bproj_tw", 1)])
def test_forward3d_columns_and_windows(oracle_mod, geom, op, B, W, H, dep, cols, cell, pz):
    _check3d(oracle_mod, geom, op, W, H, dep, cols, 20, 4, B, cell, pz)


# 64 rows that meet more slices than a step holds, 32 that do not
@pytest.mark.parametrize("rows", [33, 64, 65])
@pytest.mark.parametrize("geom,op,B", [("cone_flat", "proj", 1), ("cone_arc", "bproj_tw", 2), ("spiral", "proj", 2)])
def test_forward3d_rows_of_many_slices(oracle_mod, geom, op, B, rows):
    _check3d(oracle_mod, geom, op, 37, 44, 90, 45, rows, 5, B, pz=0.5, row=1.5)


# 16 slices a thread from 912 (tile, slab) CTAs on: 512 x 512 x 50 is past it
@pytest.mark.parametrize("W,H,dep,B", [(33, 40, 7, 3), (65, 31, 17, 1), (512, 512, 50, 1), (512, 512, 49, 3)])
@pytest.mark.parametrize("geom,op", [("cone_arc", "proj_t"), ("spiral", "bproj_w")])
def test_adjoint3d_slabs(oracle_mod, geom, op, W, H, dep, B):
    big = W > 100
    # the source outside the volume; few views of the large ones
    _check3d(oracle_mod, geom, op, W, H, dep, 300 if big else 80, 24, 2 if big else 7, B, sid=600.0 if big else 300.0)


# steps of 4 bins and 4 outputs and their remainders, groups of 4 rows, more
# outputs than a CTA's threads take at a time.  A sum of D terms in sequence
# rounds D partial sums that grow like a random walk: 2^-24 sqrt(D / 2) of it.
@pytest.mark.parametrize("D", [1, 2, 3, 4, 5, 7, 127, 128, 1023, 1025, 4098])
@pytest.mark.parametrize("rows", [1, 3, 4, 5])
def test_filter_steps(D, rows):
    from pridediff_gb300 import fbp
    rng = np.random.default_rng(D + rows)
    x, w, taps = (rng.standard_normal(s).astype(np.float32) for s in ((rows, D), (1, D), 2 * D - 1))
    out = fbp.FbpFilter.apply(*(torch.from_numpy(a).cuda() for a in (x, w, taps)))
    ref = np.stack([np.convolve(r, taps[::-1].astype(np.float64))[D - 1:2 * D - 1] for r in (x * w).astype(np.float64)])
    assert rel_l2(out.cpu().numpy(), ref) <= max(5e-7, 6e-8 * (D / 2) ** 0.5)
