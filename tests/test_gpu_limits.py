"""Calls at the limits of what the entry points accept, on the GPU.

Bars as for the same operators elsewhere: rel-L2 <= 1e-5 against the FP32
oracle in 2-D, 5e-5 in 3-D.
"""
import numpy as np
import pytest
import torch

from cases3d import spiral_source
from conftest import rel_l2
from test_gpu_2d import run as run2d
from test_gpu_3d import run as run3d
from test_gpu_splits import _check3d

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


def _apply(scan, op, opt, ang, x, slices, cluster):
    """One call through the C ABI with a forward shape asked for."""
    import ctypes
    from pridediff_gb300 import _native as N
    from pridediff_gb300 import radontorch as R
    lib, g = N.load(), N.geom2d(opt)
    a = torch.from_numpy(np.asarray(ang, np.float32)).cuda()
    xt = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    B, V, sc, opc = x.shape[0], len(ang), N.SCAN2D[scan], N.OPS[op]
    out = torch.full((B, V, g.num_det), np.nan, device="cuda")
    plan = R.plan2d(scan, g, a)
    n = lib.dd2d_apply_workspace_bytes(sc, opc, g, B, V)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    t = R.forward_tune(dict(fwd_slices=slices, fwd_cluster=cluster))
    N.check(lib.dd2d_apply_planned_tuned(sc, opc, g, plan.data_ptr(), xt.data_ptr(), out.data_ptr(), B, V, ws.data_ptr(),
                                         n, ctypes.byref(t), R._stream_ptr(a.device)), f"{scan} {op}")
    torch.cuda.synchronize()
    return out.cpu().numpy()


# Lines of which 8, 4, 2 or 1 slices fit a CTA: about 1,000, 2,750 (2,490 of
# the parallel beam with a full detector) and 3,430 pixels, the last only with
# the sums of a single CTA.
@pytest.mark.parametrize("W,D", [(1080, 700), (2480, 1984), (2790, 300), (3450, 1984), (3465, 1900), (4096, 1984)])
@pytest.mark.parametrize("scan,B", [("para", 1), ("para", 2), ("para", 3), ("flat", 9)])
def test_long_lines_in_every_shape(oracle_mod, scan, B, W, D):
    pix = 0.7 * 1080 / W
    opt = [W, 3, D, pix, pix, {"para": 1.0, "flat": 1085.6 / 595.0}[scan] * 1.1 * W * pix / D, 595.0, 1085.6, 0.1, -0.2, 0.1]
    ang = np.array([0.2, 1.4, 3.3], np.float32)
    x = np.random.default_rng(W + B).random((B, 3, W), dtype=np.float32)
    ref = oracle_mod.run2d(scan, "proj", x, ang, opt, nthreads=8)
    out = [_apply(scan, "proj", opt, ang, x, s, c) for s in (4, 1) for c in (2, 1)] + [run2d(scan, "proj", x, ang, opt)]
    assert rel_l2(out[0], ref) <= 1e-5
    for o in out[1:]:
        assert np.array_equal(o, out[0])


# A row table of 8,190 to 11,300 rows: three of them do not fit the adjoint's
# shared memory, two do.
@pytest.mark.parametrize("rows", [8100, 8191, 9000, 11300])
@pytest.mark.parametrize("geom,fwd,adj", [("cone_flat", "proj", "proj_t"), ("spiral", "bproj_tw", "bproj_w")])
def test_tall_detector(oracle_mod, geom, fwd, adj, rows):
    W, H, dep, cols, V, sid = 20, 24, 18, 12, 4, 300.0
    col, row = 5.0 * (1.0 if geom == "cone_flat" else 0.5 / sid), 60.0 / rows
    opt = [W, H, dep, cols, rows, 1.0, 1.1, 1.0, col, row, sid, 2 * sid, 0.3, -0.2]
    opt = np.array(opt + ([0.1 * col, 0.3] if geom == "spiral" else [0.4, 0.1 * col, 0.3]), np.float32)
    ang = (np.arange(V) * 2 * np.pi / V + 0.1).astype(np.float32)
    sp = spiral_source(V, 0.5, -0.25 * V) if geom == "spiral" else None
    rng = np.random.default_rng(rows)
    for op, shape in ((fwd, (1, dep, H, W)), (adj, (1, V, rows, cols))):
        x = rng.random(shape).astype(np.float32)
        ref = oracle_mod.run3d(geom, op, x, ang, opt, source_pos=sp, nthreads=8)
        assert np.any(ref)
        assert rel_l2(run3d(geom, op, x, ang, opt, sp), ref) <= 5e-5


# A 3-D workspace that starts on any address: every call works from its first
# 16-byte boundary on and stays inside the bytes it asked for.
@pytest.mark.parametrize("shift", [0, 1, 4, 8, 15])
@pytest.mark.parametrize("op,B", [("proj", 1), ("proj", 3), ("proj_t", 1), ("proj_t", 2), ("dc", 2)])
def test_workspace_at_any_address(op, B, shift):
    import ctypes
    from pridediff_gb300 import _native as N
    from pridediff_gb300 import radontorch as R
    lib, sc = N.load(), N.SCAN3D["cone_flat"]
    g = N.geom3d([30, 26, 21, 40, 18, 1.0, 1.0, 1.0, 1.6, 1.6, 300.0, 600.0, 0.0, 0.0, 0.0, 0.0, 0.0])
    V = 5
    a = torch.arange(V, dtype=torch.float32, device="cuda") * (2 * np.pi / V)
    gen = torch.Generator(device="cuda").manual_seed(3)
    vol, sino = torch.rand((B, 21, 26, 30), device="cuda", generator=gen), torch.rand((B, V, 18, 40), device="cuda", generator=gen)
    plan = R.plan3d("cone_flat", g, a)
    n = int(lib.dd3d_dc_workspace_bytes(sc, g, B, V) if op == "dc" else
            lib.dd3d_apply_workspace_bytes(sc, N.OPS[op], g, B, V))

    def call(at):
        buf = torch.full((n + 32,), 0xA5, dtype=torch.uint8, device="cuda")
        st = R._stream_ptr(a.device)
        if op == "dc":
            x, resid = vol.clone(), torch.empty_like(sino)
            N.check(lib.dd3d_dc_step(sc, g, plan.data_ptr(), x.data_ptr(), sino.data_ptr(), resid.data_ptr(),
                                     ctypes.c_float(1e-4), B, V, buf.data_ptr() + at, n, st), op)
            res = x
        else:
            src, res = (vol, torch.empty_like(sino)) if op == "proj" else (sino, torch.empty_like(vol))
            N.check(lib.dd3d_apply_planned(sc, N.OPS[op], g, plan.data_ptr(), src.data_ptr(), res.data_ptr(), B, V,
                                           buf.data_ptr() + at, n, st), op)
            word = ctypes.c_int(-1)
            assert lib.dd3d_planned_status(N.OPS[op], g, B, V, buf.data_ptr() + at, ctypes.byref(word)) == N.DD_OK
            assert word.value == N.DD_OK
        torch.cuda.synchronize()
        assert bool((buf[:at] == 0xA5).all()) and bool((buf[at + n:] == 0xA5).all())
        return res
    assert torch.equal(call(shift), call(0))


# 3-D forward, 32 columns that meet more than 64 pixels: a tile of 96 or 128
# where it holds a line's slices (20 rows), else the step's segments with
# pixels from global memory (thin slices); columns of 9 to 16 pixels, and more.
@pytest.mark.parametrize("rows,pz", [(20, 1.0), (65, 0.3)])
@pytest.mark.parametrize("cell,cols", [(2.0, 70), (2.6, 45), (3.6, 40), (7.0, 33), (11.0, 14), (14.5, 10), (25.0, 6)])
@pytest.mark.parametrize("geom,op,B", [("cone_flat", "proj", 2), ("cone_arc", "bproj_t", 1), ("spiral", "bproj_tw", 3)])
def test_forward3d_columns_of_several_pixels(oracle_mod, geom, op, B, cell, cols, rows, pz):
    _check3d(oracle_mod, geom, op, 150, 117, 40, cols, rows, 4, B, cell, pz)


# The weighted transpose's table of a line's weights: many cells a pixel, cells
# of many pixels, lines of which 8, 4, 2 and 1 slices fit beside it.
@pytest.mark.parametrize("W,H,D,cell,B", [(60, 45, 300, 0.25, 1), (45, 60, 1984, 0.04, 8), (60, 45, 9, 12.0, 4), (1, 50, 40, 1.0, 2),
                                          (890, 4, 300, 3.2, 9), (1000, 4, 300, 3.6, 9), (2500, 3, 700, 3.9, 5), (3450, 3, 1984, 1.8, 2),
                                          (4096, 3, 1984, 2.2, 2)])
@pytest.mark.parametrize("geom", ["flat", "arc"])
def test_weighted_transpose(oracle_mod, geom, W, H, D, cell, B):
    pix = 0.7 * min(1.0, 1000.0 / W)
    det = cell * pix * {"flat": 1085.6 / 595.0, "arc": 1.0 / 595.0}[geom]
    opt = [W, H, D, pix, 0.9 * pix, det, 595.0, 1085.6, 0.1, -0.2, 0.1 * det]
    ang = (np.arange(5) * 2 * np.pi / 5 + 0.1).astype(np.float32)
    x = np.random.default_rng(D).random((B, H, W), dtype=np.float32)
    ref = oracle_mod.run2d(geom, "bproj_tw", x, ang, opt, nthreads=8)
    assert np.any(ref) and rel_l2(run2d(geom, "bproj_tw", x, ang, opt), ref) <= 1e-5


# Lines that leave 8 slices no room beside that table: groups of 8 weigh each
# overlap, the slices left over (none to 7) take the table's weights.
@pytest.mark.parametrize("W,H,D,B", [(950, 4, 200, 8), (4, 950, 420, 16), (1000, 5, 650, 9), (930, 3, 900, 11), (900, 7, 1000, 15)])
@pytest.mark.parametrize("geom", ["flat", "arc"])
def test_weighted_transpose_groups_of_eight(oracle_mod, geom, W, H, D, B):
    pix = 0.7 * 1000.0 / max(W, H)
    det = 1200.0 / D * pix * {"flat": 1085.6 / 595.0, "arc": 1.0 / 595.0}[geom]
    opt = [W, H, D, pix, 0.9 * pix, det, 595.0, 1085.6, 0.1, -0.2, 0.1 * det]
    ang = (np.arange(5) * 2 * np.pi / 5 + 0.1).astype(np.float32)
    x = np.random.default_rng(D).random((B, H, W), dtype=np.float32)
    ref = oracle_mod.run2d(geom, "bproj_tw", x, ang, opt, nthreads=8)
    out = run2d(geom, "bproj_tw", x, ang, opt)
    assert np.any(ref) and rel_l2(out, ref) <= 1e-5
    for b in (0, 7, B - 1):
        assert rel_l2(run2d(geom, "bproj_tw", x[b:b + 1], ang, opt)[0], out[b]) <= 2e-6   # the same terms, their rounding aside


# 2-D forward, bins of more than four pixels: 1 to 32 lanes a bin and up to 4
# passes of 256 lanes; each slice as it is alone, whatever the group it is in.
@pytest.mark.parametrize("W,H,D,cell", [(150, 97, 3, 45.0), (150, 97, 8, 20.0), (260, 130, 16, 17.0), (200, 150, 32, 7.0), (200, 97, 40, 5.2),
                                        (300, 64, 100, 4.1), (900, 40, 100, 9.3), (1100, 30, 180, 6.5), (1050, 20, 255, 4.3), (90, 70, 1, 60.0)])
@pytest.mark.parametrize("geom,op", [("para", "proj"), ("flat", "proj"), ("arc", "bproj_t"), ("flat", "bproj_tw")])
def test_wide_bins(oracle_mod, geom, op, W, H, D, cell):
    pix = 0.5
    det = cell * pix * {"para": 1.0, "flat": 1085.6 / 595.0, "arc": 1.0 / 595.0}[geom]
    opt = [W, H, D, pix, 0.9 * pix, det, 595.0, 1085.6, 0.1, -0.2, 0.1 * det]
    ang = (np.arange(5) * 2 * np.pi / 5 + 0.1).astype(np.float32)
    x = np.random.default_rng(D).random((9, H, W), dtype=np.float32)
    ref = oracle_mod.run2d(geom, op, x, ang, opt, nthreads=8)
    out = run2d(geom, op, x, ang, opt)
    assert np.any(ref) and rel_l2(out, ref) <= 1e-5
    for B in (1, 2, 4, 5):
        assert np.array_equal(run2d(geom, op, x[:B], ang, opt), out[:B])


@pytest.mark.parametrize("scan", ["flat", "para"])
def test_uneven_batch_of_wide_and_narrow_bins(scan):
    import pridediff_gb300 as P
    from pridediff_gb300.batch import UnevenBatch2d
    sizes, dets, batch = [(64, 48), (150, 70), (96, 96), (200, 40)], [100, 20, 96, 12], [1, 3, 2, 5]
    cells = [0.66 * c * (1085.6 / 595.0 if scan == "flat" else 1.0) for c in (1.0, 9.0, 1.3, 19.0)]
    projs = [P.projector2d(s, d, 0.66, c, 595.0, 1085.6, scan_type=scan).cuda() for s, d, c in zip(sizes, dets, cells)]
    angs = [torch.arange(v, dtype=torch.float32, device="cuda") * (2 * np.pi / v) for v in (9, 20, 33, 7)]
    ub = UnevenBatch2d(projs, angs, batch)
    g = torch.Generator(device="cuda").manual_seed(5)
    xs = [torch.rand(s, device="cuda", generator=g) for s in ub.img_shapes]
    for p, a, x, y in zip(projs, angs, xs, ub.unpack_sinos(ub.forward(ub.pack(xs)))):
        # the two forwards' roundings, each within 1e-5 of exact arithmetic
        assert rel_l2(y.cpu().numpy(), p.projection(x, a).cpu().numpy()) <= 2e-5


# Parallel adjoint: a line by one CTA (the lines fill the chip and the tables
# leave room for two CTAs an SM) or by a cluster of four, with the same bits --
# the uneven batch always takes the cluster.  1 to 4 pixels a thread, fewer
# views than parts.
@pytest.mark.parametrize("W,H,D,V,B", [(300, 270, 1200, 6, 4), (300, 270, 1200, 1, 4), (270, 560, 1300, 9, 5), (249, 300, 1800, 3, 9),
                                       (900, 300, 1250, 4, 8), (300, 40, 1200, 5, 4)])
def test_parallel_adjoint_by_one_and_four(oracle_mod, W, H, D, V, B):
    import pridediff_gb300 as P
    from pridediff_gb300.batch import UnevenBatch2d
    proj = P.projector2d((W, H), D, 0.7, 0.7 * 1.3 * W / D, 595.0, 1085.6, scan_type="para").cuda()
    ang = torch.arange(V, dtype=torch.float32, device="cuda") * (np.pi / V) + 0.3
    y = torch.randn((B, 1, V, D), device="cuda", generator=torch.Generator(device="cuda").manual_seed(W))
    out = proj.projection_t(y, ang)
    ub = UnevenBatch2d([proj], [ang], [B])
    assert torch.equal(ub.adjoint(y.reshape(-1)).reshape(out.shape), out)
    ref = oracle_mod.run2d("para", "proj_t", y[:, 0].cpu().numpy(), ang.cpu().numpy(), proj.options.cpu().numpy(), nthreads=8)
    assert rel_l2(out[:, 0].cpu().numpy(), ref) <= 1e-5


# Stages given up for a third CTA on an SM (parallel beam, 2 records a
# producer): 8, 7, 6 and 5 stages of one and two slices, both cluster sizes.
@pytest.mark.parametrize("W,D", [(512, 736), (600, 800), (700, 900), (900, 1000)])
@pytest.mark.parametrize("scan,B", [("para", 1), ("para", 2), ("flat", 1)])
def test_forward_stages(oracle_mod, scan, B, W, D):
    pix = 0.5
    opt = [W, 24, D, pix, pix, {"para": 1.0, "flat": 1085.6 / 595.0}[scan] * 1.1 * W * pix / D, 595.0, 1085.6, 0.1, -0.2, 0.1]
    ang = (np.arange(5) * 2 * np.pi / 5 + 0.1).astype(np.float32)
    x = np.random.default_rng(W + B).random((B, 24, W), dtype=np.float32)
    ref = oracle_mod.run2d(scan, "proj", x, ang, opt, nthreads=8)
    out = [_apply(scan, "proj", opt, ang, x, s, c) for s in (4, 1) for c in (2, 1)]
    assert rel_l2(out[0], ref) <= 1e-5
    for o in out[1:]:
        assert np.array_equal(o, out[0])
