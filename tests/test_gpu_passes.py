"""The 2-D forward at the edges of its detector passes (256 bins; 248 of the arc
fan's prefix sums), the arc fan across batch sizes, and the timeout path of the
kernels that tests/test_gpu_timeouts.py does not reach.

Bars as for the same operators elsewhere: rel-L2 <= 1e-5 against the FP32
oracle.
"""
import ctypes

import numpy as np
import pytest
import torch

from conftest import rel_l2
from test_gpu_2d import run as run2d
from test_gpu_splits import _check2d, _turn
from test_gpu_timeouts import _expect_timeout, _stream, waitlib   # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu


# the last bin of a pass and the first of the next, in every class of passes
@pytest.mark.parametrize("D", [256, 257, 512, 513, 768, 769, 1024, 1025, 1984])
@pytest.mark.parametrize("geom,op,B", [("para", "proj", 1), ("para", "bproj_t", 4), ("flat", "proj", 2), ("flat", "bproj_tw", 8),
                                       ("arc", "proj", 4), ("arc", "bproj_t", 1)])
def test_overlap_passes(oracle_mod, geom, op, B, D):
    _check2d(oracle_mod, geom, op, 40, 57, D, _turn(5), B, 70.0 / D, seed=D)


# the arc fan's projection of one and two slices: by prefix sums, 8 warps of 31
# bins a pass, or by overlaps where those would round too much (1090 x 5 with
# many cells).  (1 x 9 pixels stop at 993 cells: of 1,984 a boundary's last bit,
# which device and host trigonometry round apart, is 1e-5 of a sum.)
@pytest.mark.parametrize("W,H,D", [(w, h, d) for w, h in ((40, 57), (1, 9), (1090, 5))
                                   for d in (1, 247, 248, 249, 496, 497, 744, 745, 992, 993, 1984) if h != 9 or d < 1984])
@pytest.mark.parametrize("B", [1, 2])
def test_prefix_passes(oracle_mod, W, H, B, D):
    _check2d(oracle_mod, "arc", "proj", W, H, D, _turn(5), B, (1.7 if W < 1000 else 0.9) * max(W, H) / D, seed=D)


# A slice of an arc fan is projected by prefix sums alone or in a pair, by
# overlaps in larger groups: equal bits within either, and between them the
# prefix sums' rounding (each boundary's to 2^-25 of a line's integral, N
# pixels: 2^-25 N sqrt(2 / L) of a sum over L lines, 5e-7 here; four times that).
# A data-consistency block of any size is the composition of its operators.
def test_arc_slices_across_batch_sizes():
    import pridediff_gb300 as P
    from pridediff_gb300.fidelity import FidelityModule
    proj = P.projector2d(128, 192, 2.64, 1.2858 * 4, 595.0, 1085.6, scan_type="arc").cuda().requires_grad_(False)
    ang = torch.arange(180, dtype=torch.float32, device="cuda") * (2 * np.pi / 180)
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.rand((8, 1, 128, 128), device="cuda", generator=g)
    y = torch.rand((8, 1, 180, 192), device="cuda", generator=g)
    block = FidelityModule(proj, ang, adjoint="fbp").cuda().requires_grad_(False)
    block.weight.fill_(0.3)
    one = torch.cat([proj.projection(x[i:i + 1], ang) for i in range(8)])
    many = proj.projection(x, ang)
    assert rel_l2(many.cpu().numpy(), one.cpu().numpy()) <= 2e-6
    for n in (1, 2, 3, 4, 5, 8):
        a = proj.projection(x[:n], ang)
        assert torch.equal(a, (one if n <= 2 else many)[:n])
        assert torch.equal(block(x[:n], y[:n]), x[:n] - block.weight * proj.filtered_backprojection(a - y[:n], ang))


@pytest.mark.parametrize("B", [1, 2])
def test_prefix_forward_timeout(waitlib, B):   # noqa: F811
    N, lib, word = waitlib
    g = N.Geom2d(64, 48, 300, 1.0, 1.0, 0.4 / 500.0, 500.0, 1000.0, 0.0, 0.0, 0.0)
    V, sc, opc = 24, N.SCAN2D["arc"], N.OPS["proj"]
    ang = torch.arange(V, dtype=torch.float32, device="cuda") * (2 * np.pi / V)
    x, out = torch.rand((B, 48, 64), device="cuda"), torch.zeros((B, V, 300), device="cuda")
    n = lib.dd2d_workspace_bytes(sc, opc, ctypes.byref(g), B, V)
    ws = torch.zeros(n, dtype=torch.uint8, device="cuda")
    assert lib.dd2d_apply(sc, opc, ctypes.byref(g), x.data_ptr(), out.data_ptr(), ang.data_ptr(), B, V, ws.data_ptr(), n,
                          _stream()) == N.DD_OK
    _expect_timeout(N, word, lambda p: lib.dd2d_status(sc, opc, ctypes.byref(g), B, V, ws.data_ptr(), p))


@pytest.mark.parametrize("cluster", [1, 2])
def test_parallel_uneven_batch_timeouts(waitlib, cluster):   # noqa: F811
    N, lib, word = waitlib
    sizes = [(64, 24, 80, 1), (48, 16, 72, 3), (96, 20, 6, 2)]   # the last with wide bins
    inst = (N.Instance2d * len(sizes))()
    angs = []
    for i, (n, V, D, b) in enumerate(sizes):
        inst[i].geom = N.Geom2d(n, n, D, 1.0, 1.0, 1.2 * n / D, 500.0, 1000.0, 0.0, 0.0, 0.0)
        inst[i].num_view, inst[i].batch = V, b
        angs.append(torch.arange(V, dtype=torch.float32, device="cuda") * (np.pi / V))
    sc, tune = N.SCAN2D["para"], N.Tune2d(0, 1, 0, 0, cluster)
    pb, wb = lib.dd2d_batch_plan_bytes(sc, inst, len(sizes)), lib.dd2d_batch_workspace_bytes(sc, inst, len(sizes))
    plan, ws = (torch.zeros(k, dtype=torch.uint8, device="cuda") for k in (pb, wb))
    ptrs = (ctypes.c_void_p * len(sizes))(*[a.data_ptr() for a in angs])
    assert lib.dd2d_batch_plan(sc, inst, len(sizes), ptrs, plan.data_ptr(), pb, ctypes.byref(tune), _stream()) == N.DD_OK
    img, sino = sum(b * n * n for n, _, _, b in sizes), sum(b * V * D for _, V, D, b in sizes)
    for op, nin, nout in (("proj", img, sino), ("proj_t", sino, img)):
        x, out = torch.rand(nin, device="cuda"), torch.zeros(nout, device="cuda")
        assert lib.dd2d_batch_apply(sc, N.OPS[op], inst, len(sizes), plan.data_ptr(), x.data_ptr(), out.data_ptr(),
                                    ws.data_ptr(), wb, ctypes.byref(tune), _stream()) == N.DD_OK
        _expect_timeout(N, word, lambda p: lib.dd2d_batch_status(sc, inst, len(sizes), ws.data_ptr(), p))


# the parallel adjoint by one CTA a line, and the wide bins' forward
@pytest.mark.parametrize("op,W,D", [("proj_t", 300, 1200), ("proj", 300, 20)])
def test_parallel_timeouts(waitlib, op, W, D):   # noqa: F811
    N, lib, word = waitlib
    H, V, B, sc, opc = 280, 6, 4, N.SCAN2D["para"], N.OPS[op]
    g = N.Geom2d(W, H, D, 1.0, 1.0, 1.2 * W / D, 500.0, 1000.0, 0.0, 0.0, 0.0)
    ang = torch.arange(V, dtype=torch.float32, device="cuda") * (np.pi / V) + 0.2
    img, sino = (B, H, W), (B, V, D)
    x, out = torch.rand(img if op == "proj" else sino, device="cuda"), torch.zeros(sino if op == "proj" else img, device="cuda")
    n = lib.dd2d_workspace_bytes(sc, opc, ctypes.byref(g), B, V)
    ws = torch.zeros(n, dtype=torch.uint8, device="cuda")
    assert lib.dd2d_apply(sc, opc, ctypes.byref(g), x.data_ptr(), out.data_ptr(), ang.data_ptr(), B, V, ws.data_ptr(), n,
                          _stream()) == N.DD_OK
    _expect_timeout(N, word, lambda p: lib.dd2d_status(sc, opc, ctypes.byref(g), B, V, ws.data_ptr(), p))


def test_results_after_the_timeouts(waitlib, oracle_mod):   # noqa: F811
    ang = _turn(7).astype(np.float32)
    opt = [40, 31, 60, 0.7, 0.7, 0.9, 595.0, 1085.6, 0.0, 0.0, 0.0]
    x = np.random.default_rng(1).random((2, 31, 40), dtype=np.float32)
    assert rel_l2(run2d("para", "proj", x, ang, opt), oracle_mod.run2d("para", "proj", x, ang, opt, nthreads=4)) <= 1e-5
