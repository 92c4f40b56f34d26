"""What a user of this projector has it do, as cases that can be timed and compared.

A case names a scan geometry, its sizes and an operation: ``project`` (A x),
``adjoint`` (A^T y), ``step`` (loss ||A x - y||^2 and its gradient through
autograd), ``fbp`` (filtered back-projection), ``fidelity`` (the
data-consistency block of a network, forward and backward) and ``dc`` (one
data-consistency step of an uneven batch).  ``exact`` restates each of them in
64 bits with plain torch: distance-driven projection is the overlap of pixel
(voxel) footprints with detector cells on a projection axis, so each view is a
resampling of the running integral of every image line (detector row) at the
boundaries of the cells (pixels).
"""
import math

import numpy as np
import torch

import pridediff_gb300 as P
from pridediff_gb300.batch import UnevenBatch2d
from pridediff_gb300.fidelity import FidelityModule

DEV = "cuda"


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call of an interactive or unit-test-like use: launches and host path
        dict(name="para_64_project_1", scan="para", op="project", w=64, h=64, dets=95, views=60, batch=1, shift=False),
        # one training / reconstruction step on the small CT configuration
        dict(name="para_256_step_1", scan="para", op="step", w=256, h=256, dets=367, views=180, batch=1, shift=False),
        # simulating the scan of a single slice
        dict(name="flat_512_project_1", scan="flat", op="project", w=512, h=512, dets=736, views=720, batch=1,
             shift=False),
        # the main workload: loss and gradient of a batch of slices
        dict(name="flat_512_step_16", scan="flat", op="step", w=512, h=512, dets=736, views=720, batch=16,
             shift=False),
        # back-projection of a few slices on an odd, off-centre grid with a shifted detector
        dict(name="flat_odd_adjoint_3", scan="flat", op="adjoint", w=403, h=331, dets=517, views=391, batch=3,
             shift=True),
        # FBP reconstruction of a few slices from an arc detector
        dict(name="arc_512_fbp_4", scan="arc", op="fbp", w=512, h=512, dets=768, views=720, batch=4, shift=False),
        # a diffusion model's data-consistency block in training: forward and backward
        dict(name="arc_512_fidelity_2", scan="arc", op="fidelity", w=512, h=512, dets=768, views=720, batch=2,
             shift=False),
        # data consistency of many slices of different scanners at once
        dict(name="uneven_24_dc", scan="uneven", op="dc", instances=24, pick=2024),
        # the cone-beam training step: the largest case
        dict(name="cone_flat_256_step_2", scan="cone_flat", op="step", w=256, h=256, depth=256, dets=512, rows=384,
             views=360, batch=2, shift=False),
        # FDK-like reconstruction of a small off-centre volume from an arc detector, odd sizes
        dict(name="cone_arc_odd_fbp_1", scan="cone_arc", op="fbp", w=141, h=119, depth=75, dets=201, rows=99,
             views=123, batch=1, shift=True),
        # a turn of a helical scan of a full-size volume: simulation ...
        dict(name="spiral_512_project_1", scan="spiral", op="project", w=512, h=512, depth=128, dets=736, rows=64,
             views=1140, batch=1, shift=False),
        # ... and its gradient
        dict(name="spiral_512_adjoint_1", scan="spiral", op="adjoint", w=512, h=512, depth=128, dets=736, rows=64,
             views=1140, batch=1, shift=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    scan = rng.choice(["para", "flat", "flat", "arc", "arc", "uneven", "cone_flat", "cone_arc", "spiral"])
    if scan == "uneven":
        return dict(scan="uneven", op="dc", instances=_log(rng, 2, 24), pick=rng.randrange(1 << 20))
    shift = rng.random() < 0.5
    if scan in ("para", "flat", "arc"):
        w = _log(rng, 64, 512)
        h = w if rng.random() < 0.5 else max(64, min(512, int(w * rng.uniform(0.7, 1.4))))
        return dict(scan=scan, op=rng.choice(["project", "adjoint", "step", "fbp"] + ["fidelity"] * (scan == "arc")),
                    w=w, h=h, dets=int(max(w, h) * rng.uniform(0.8, 1.5)), views=_log(rng, 60, 720),
                    batch=_log(rng, 1, 16), shift=shift)
    if scan == "spiral":
        w = _log(rng, 64, 512)
        return dict(scan=scan, op=rng.choice(["project", "adjoint"]), w=w, h=w, depth=_log(rng, 16, 128),
                    dets=int(w * rng.uniform(1.0, 1.5)), rows=rng.choice([16, 32, 48, 64]),
                    views=_log(rng, 150, 1140), batch=1 if w > 256 else rng.choice([1, 2]), shift=shift)
    w = _log(rng, 64, 224)
    h = w if rng.random() < 0.5 else int(w * rng.uniform(0.8, 1.2))
    return dict(scan=scan, op=rng.choice(["project", "adjoint", "step", "fbp"]), w=w, h=h,
                depth=int(w * rng.uniform(0.4, 1.0)), dets=int(w * rng.uniform(1.2, 2.0)),
                rows=int(w * rng.uniform(0.8, 1.5)), views=_log(rng, 60, 240), batch=rng.choice([1, 2]), shift=shift)


# ---------------------------------------------------------------------------
# Geometries
# ---------------------------------------------------------------------------
def _geometry(case):
    """The scanner of a case: what its projector is built from, and its views."""
    s, n, w = case["scan"], case["dets"], case["w"]
    k = 1.0 if case["shift"] else 0.0
    if s == "para":   # 1 mm cells over 180 degrees
        return dict(pix=(1.0, 1.0), det=1.0, iso=500.0, sdd=1000.0, pixshift=(1.3 * k, -0.7 * k), binshift=0.25 * k,
                    arc=math.pi)
    if s == "flat":   # 338 mm field, 946 mm detector
        return dict(pix=(0.66 * 512 / w,) * 2, det=1.2858 * 736 / n, iso=595.0, sdd=1085.6,
                    pixshift=(1.3 * k, -0.7 * k), binshift=0.25 * k * 1.2858 * 736 / n, arc=2 * math.pi)
    if s == "arc":    # the same field, 768 cells on an arc
        return dict(pix=(0.66 * 512 / w,) * 2, det=1.2858 * 768 / n, iso=595.0, sdd=1085.6,
                    pixshift=(1.3 * k, -0.7 * k), binshift=0.25 * k * 1.2858 * 768 / n, arc=2 * math.pi)
    if s == "spiral":   # 338 mm field, 64 mm of 1 mm rows, 1152 views a turn
        return dict(pix=(0.66 * 512 / w, 0.66 * 512 / w, 1.0), det=(1.2858 * 736 / n, 64.0 / case["rows"]),
                    iso=595.0, sdd=1085.6, pixshift=(1.3 * k, -0.7 * k), binshift=(0.25 * k * 1.2858 * 736 / n, 0.0),
                    arc=2 * math.pi * case["views"] / 1152)
    p = 256.0 / w     # 256 mm field, 512 mm x 384 mm detector
    return dict(pix=(p, p, p), det=(512.0 / n, 384.0 / case["rows"]), iso=500.0, sdd=1000.0,
                pixshift=(1.3 * k, -0.7 * k, 0.4 * k), binshift=(0.25 * k * 512.0 / n, 0.3 * k), arc=2 * math.pi)


def _views(case, g):
    return (np.arange(case["views"]) * (g["arc"] / case["views"])).astype(np.float32)


def _table(case):
    """The helix: pitch 1 (a detector height at the axis per turn), centred on the volume."""
    v = case["views"]
    step = 64.0 * 595.0 / 1085.6 / 1152
    sp = np.zeros((4, v), np.float32)
    sp[0] = (step * (np.arange(v) - (v - 1) / 2)).astype(np.float32)
    return sp


def _projector(case, g):
    kind = {"para": "para", "flat": "flat", "arc": "arc", "cone_flat": "flat", "cone_arc": "arc", "spiral": "arc"}
    if "depth" not in case:
        p = P.projector2d((case["w"], case["h"]), case["dets"], g["pix"], g["det"], g["iso"], g["sdd"],
                          pixshift=g["pixshift"], binshift=g["binshift"], scan_type=kind[case["scan"]])
    else:
        cls = P.projectorsp if case["scan"] == "spiral" else P.projector3d
        p = cls((case["w"], case["h"], case["depth"]), (case["dets"], case["rows"]), g["pix"], g["det"], g["iso"],
                g["sdd"], pixshift=g["pixshift"], binshift=g["binshift"], scan_type=kind[case["scan"]])
    # the network's projector is not trained here
    return p.requires_grad_(False).to(DEV)


_SIZES = dict(size=[256, 384, 512], views=[360, 576, 720], dets=[368, 512, 736])


def _instances(case):
    """The slices of an uneven batch, drawn from three image sizes, view counts and detectors."""
    rng = np.random.default_rng(case["pick"])
    out = []
    for _ in range(case["instances"]):
        n, v, d = (int(rng.choice(_SIZES[k])) for k in ("size", "views", "dets"))
        out.append(dict(scan="flat", w=n, h=n, dets=d, views=v, batch=1, shift=False))
    return out


def _instance_geometry():
    """An uneven batch's scanner: 0.66 mm pixels and 1.2858 mm cells whatever their number."""
    return dict(pix=(0.66, 0.66), det=1.2858, iso=595.0, sdd=1085.6, pixshift=(0.0, 0.0), binshift=0.0,
                arc=2 * math.pi)


# ---------------------------------------------------------------------------
# Inputs: phantoms of random ellipses (attenuation up to 0.04 / mm) and
# sinograms of random discs (line integrals up to about 8) with noise
# ---------------------------------------------------------------------------
def _phantom(shape, gen):
    b, dims = shape[0], shape[2:]
    axes = [torch.linspace(-1, 1, n, device=DEV).view([-1 if i == a else 1 for i in range(len(dims))])
            for a, n in enumerate(dims)]
    img = torch.zeros(shape, device=DEV)
    for i in range(b):
        for _ in range(8):
            r = torch.rand(2 * len(dims) + 1, generator=gen, device=DEV)
            q = sum(((x - (1.4 * r[a] - 0.7)) / (0.08 + 0.35 * r[len(dims) + a])) ** 2 for a, x in enumerate(axes))
            img[i, 0] += (q <= 1) * r[-1]
    return img.clamp_(0, 1).mul_(0.04)


def _sinogram(shape, gen):
    b, v, d = shape[0], shape[2], shape[-1]
    ang = torch.arange(v, device=DEV) * (2 * math.pi / v)
    u = torch.linspace(-1, 1, d, device=DEV)
    out = torch.zeros((b, 1, v, d), device=DEV)
    for i in range(b):
        for _ in range(6):
            r = torch.rand(4, generator=gen, device=DEV)
            c = 0.5 * r[0] * torch.cos(ang + 6.28 * r[1])[:, None]
            out[i, 0] += 3.0 * r[3] * (1 - ((u - c) / (0.06 + 0.25 * r[2])) ** 2).clamp_(min=0).sqrt_()
    if len(shape) == 5:
        row = torch.linspace(-1, 1, shape[3], device=DEV)
        out = out[:, :, :, None, :] * (1 - 0.5 * row ** 2)[:, None]
    return out + 0.02 * torch.randn(shape, generator=gen, device=DEV)


def _shapes(case):
    lead = (case["batch"], 1)
    if "depth" in case:
        return lead + (case["depth"], case["h"], case["w"]), lead + (case["views"], case["rows"], case["dets"])
    return lead + (case["h"], case["w"]), lead + (case["views"], case["dets"])


_ETA = 4e-6      # below 2 / lambda_max(A^T A) of the largest instance
_WEIGHT = 0.3    # the block's learned weight


def _inputs(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)
    if case["scan"] == "uneven":
        parts = _instances(case)
        return [_phantom(_shapes(c)[0], gen) for c in parts], [_sinogram(_shapes(c)[1], gen) for c in parts]
    img, sino = _shapes(case)
    d = {}
    if case["op"] in ("project", "step", "fidelity"):
        d["x"] = _phantom(img, gen)
    if case["op"] in ("adjoint", "step", "fbp", "fidelity"):
        d["y"] = _sinogram(sino, gen)
    if case["op"] == "fidelity":
        d["g"] = torch.randn(img, generator=gen, device=DEV)
    return d


def prepare(case, seed):
    if case["scan"] == "uneven":
        xs, ys = _inputs(case, seed)
        g = _instance_geometry()
        parts = _instances(case)
        batch = UnevenBatch2d([_projector(c, g) for c in parts],
                              [torch.from_numpy(_views(c, g)).to(DEV) for c in parts])
        return dict(op="dc", batch=batch, x=batch.pack(xs), y=batch.pack(ys))
    g = _geometry(case)
    s = dict(_inputs(case, seed), op=case["op"], proj=_projector(case, g),
             views=(torch.from_numpy(_views(case, g)).to(DEV),))
    if case["scan"] == "spiral":
        s["views"] += (torch.from_numpy(_table(case)).to(DEV),)
    if case["op"] in ("step", "fidelity"):
        s["x"].requires_grad_(True)
    if case["op"] == "fidelity":
        s["block"] = FidelityModule(s["proj"], s["views"][0], adjoint="fbp").to(DEV)
        with torch.no_grad():
            s["block"].weight.fill_(_WEIGHT)
    return s


def run(s):
    op = s["op"]
    if op == "project":
        return s["proj"].projection(s["x"], *s["views"])
    if op == "adjoint":
        return s["proj"].projection_t(s["y"], *s["views"])
    if op == "fbp":
        return s["proj"].filtered_backprojection(s["y"], *s["views"])
    if op == "dc":
        return s["batch"].dc_step(s["x"], s["y"], _ETA)
    if op == "step":
        s["x"].grad = None
        p = s["proj"].projection(s["x"], *s["views"])
        loss = ((p - s["y"]) ** 2).sum()
        loss.backward()
        return [p.detach(), s["x"].grad]
    s["x"].grad = s["block"].weight.grad = None
    out = s["block"](s["x"], s["y"])
    out.backward(s["g"])
    return [out.detach(), s["x"].grad, s["block"].weight.grad]


# ---------------------------------------------------------------------------
# What a pass cannot do without: inputs read once, outputs written once, and a
# multiply-add for each overlap of a pixel (voxel) with a detector cell
# ---------------------------------------------------------------------------
def work(case):
    if case["scan"] == "uneven":
        parts = [work(dict(c, op="dc")) for c in _instances(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    img, sino = (math.prod(s) for s in _shapes(case))
    lines, v, b = (case["w"] + case["h"]) / 2, case["views"], case["batch"]
    if "depth" not in case:
        cells = b * v * lines * (lines + case["dets"])
    else:
        seen = case["depth"]
        if case["scan"] == "spiral":   # the slices a view's cone meets, on the mean
            seen = min(seen, 1.1 * 64 * 595.0 / 1085.6)
        cells = b * v * lines * (lines * seen + case["dets"] * case["rows"])
    passes = {"project": 1, "adjoint": 1, "fbp": 1, "step": 2, "dc": 2, "fidelity": 4}[case["op"]]
    touched = {"project": img + sino, "adjoint": img + sino, "fbp": img + sino, "step": 2 * img + 2 * sino,
               "dc": 2 * img + sino, "fidelity": 4 * img + sino}[case["op"]]
    flops = 2 * cells * passes
    if case["op"] in ("fbp", "fidelity"):   # the ramp filter, by the fastest known method
        n = 4 * case["dets"]
        flops += sino / case["dets"] * 5 * n * math.log2(n) * (2 if case["op"] == "fidelity" else 1)
    return {"bytes": 4.0 * touched, "flops": float(flops)}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
def _at(table, q):
    """Piecewise linear `table` (..., N + 1) over 0 .. N at q (broadcast), clamped to its ends."""
    n = table.shape[-1] - 1
    q = q.clamp(0, n)
    i = q.floor().clamp(max=max(n - 1, 0))
    f = q - i
    i = i.long().expand(table.shape[:-1] + q.shape[-1:])
    a = table.gather(-1, i)
    return a + f * (table.gather(-1, i + 1) - a)


def _running(x, dim=-1):
    """Running sums along `dim`, a zero in front."""
    z = torch.zeros_like(x.narrow(dim, 0, 1))
    return torch.cat([z, x.cumsum(dim)], dim)


class _Exact:
    """A scanner in 64 bits: `project`, `adjoint` and the weighted back-projection."""

    def __init__(self, case, g, views=None, table=None):
        f = lambda v: float(np.float32(v))   # noqa: E731  (a user's numbers reach the framework as float32)
        self.c, self.scan = case, case["scan"]
        self.w, self.h, self.n = case["w"], case["h"], case["dets"]
        self.sx, self.sy = f(g["pix"][0]), f(g["pix"][1])
        self.px, self.py = f(g["pixshift"][0]), f(g["pixshift"][1])
        self.iso, self.sdd = f(g["iso"]), f(g["sdd"])
        self.volume = "depth" in case
        det = g["det"][0] if self.volume else g["det"]
        bins = g["binshift"][0] if self.volume else g["binshift"]
        self.fan_arc = self.scan in ("arc", "cone_arc", "spiral")
        if self.fan_arc:
            det, bins = det / g["sdd"], bins / g["sdd"]
        self.det, self.bins = f(det), f(bins)
        self.views = views
        if self.volume:
            self.depth, self.rows = case["depth"], case["rows"]
            self.sz, self.drow = f(g["pix"][2]), f(g["det"][1])
            self.pz = f(g["pixshift"][2]) if len(g["pixshift"]) > 2 else 0.0
            self.rshift = f(g["binshift"][1])
            self.table = table

    def t(self, v):
        return torch.as_tensor(v, dtype=torch.float64, device=DEV)

    def view(self, v):
        """Geometry of view v on its projection axis: which axis, the cell boundaries in ascending order, the lines."""
        a32 = torch.tensor(self.views[v], dtype=torch.float32, device=DEV)
        a = float(self.views[v])
        if self.volume:    # the axis is chosen by the single-precision cosine
            c32 = float(torch.cos(a32))
        else:
            c32 = float(np.float32(math.cos(a)))
        s, c = math.sin(a), math.cos(a)
        xb = bool(np.float32(c32) * np.float32(c32) > np.float32(0.5))
        flip = c < 0 if xb else s < 0
        n = self.n
        k = torch.arange(n + 1, dtype=torch.float64, device=DEV) - n / 2
        kk = -k if flip else k
        d = dict(xb=xb, flip=flip, s=s, c=c)
        sx, sy = -s * self.iso, c * self.iso
        mid = (kk[:-1] + kk[1:]) / 2
        if self.scan == "para":
            d["d"] = (kk * self.det + self.bins) / (c if xb else s)
        elif not self.fan_arc:
            u = (kk * self.det + self.bins) * self.iso / self.sdd
            x, y = u * c, u * s
            d["d"] = (sx * y - sy * x) / (y - sy) if xb else (sy * x - sx * y) / (x - sx)
            d["cell"] = self.det * self.iso / self.sdd
            um = (mid * self.det + self.bins) * self.iso / self.sdd
            cen = um * (s if xb else c)
        else:
            t = torch.tan(kk * self.det + self.bins + a)
            d["d"] = sx + sy * t if xb else sy + sx / t
            d["cell"] = self.det * self.iso
            am = mid * self.det + self.bins + a
            cen = -torch.cos(am) * self.sdd + sy if xb else torch.sin(am) * self.sdd + sx
        d["src"], d["srcxy"] = (sy if xb else sx), (sx, sy)
        if self.volume:
            d["mag"] = d["src"] / (d["src"] - cen)
        # walked lines: rows top down, or columns; pixel boundaries p0 + j * pitch
        nl, npix = (self.h, self.w) if xb else (self.w, self.h)
        i = torch.arange(nl, dtype=torch.float64, device=DEV)
        line = (nl / 2 - i - 0.5) * self.sy + self.py if xb else (i - nl / 2 + 0.5) * self.sx + self.px
        lo, hi = ((-npix / 2 * self.sx + self.px, npix / 2 * self.sx + self.px) if xb else
                  (-npix / 2 * self.sy + self.py, npix / 2 * self.sy + self.py))
        if self.scan == "para":
            off = line * (s / c if xb else c / s)
            d["p0"], d["pitch"] = off + lo, torch.full_like(line, self.sx if xb else self.sy)
        else:
            oth = sx if xb else sy          # the source's coordinate along the axis
            den = line - d["src"]
            b0, b1 = (oth * line - d["src"] * lo) / den, (oth * line - d["src"] * hi) / den
            d["p0"], d["pitch"] = b0, (b1 - b0) / npix
            d["m"] = -d["src"] / den
        d["line"], d["npix"] = line, npix
        # scale of a cell: chord length per area
        other = self.sy if xb else self.sx
        w = d["d"][1:] - d["d"][:-1]
        if self.scan == "para":
            d["scale"] = torch.full_like(w, other / self.det)
        elif not self.volume:
            m = (d["d"][1:] + d["d"][:-1]) / 2 - (sx if xb else sy)
            d["scale"] = other / w / (abs(d["src"]) / torch.sqrt(m * m + d["src"] ** 2))
        else:
            ctr = float(self.table[0, v]) if self.scan == "spiral" else 0.0
            r = (torch.arange(self.rows + 1, dtype=torch.float64, device=DEV) - self.rows / 2) * self.drow + self.rshift
            if self.scan == "cone_flat":
                r = r * self.iso / self.sdd
            z = d["mag"][:, None] * r + ctr            # (C, R + 1): row boundaries on the axis plane
            d["z"] = z
            m = (d["d"][1:] + d["d"][:-1]) / 2 - (sx if xb else sy)
            # the obliquity uses the row's height on the axis plane itself
            zm = (z[:, 1:] + z[:, :-1]) / 2
            q = m[:, None] ** 2 + zm ** 2 + d["src"] ** 2
            d["scale"] = (other / (w[:, None] * (z[:, 1:] - z[:, :-1])) * torch.sqrt(q) / abs(d["src"])).T  # (R, C)
            z0, z1 = -self.depth / 2 * self.sz + self.pz, self.depth / 2 * self.sz + self.pz
            d["z0"] = d["m"] * (z0 - ctr) + ctr
            d["zpitch"] = d["m"] * (z1 - z0) / self.depth
        return d

    def lines(self, x):
        """Images (.., H, W) as walked lines of either kind: rows, and columns from the bottom row up."""
        return x, x.flip(-2).transpose(-1, -2).contiguous()

    def project(self, x):
        x = x.double()[:, 0]
        out = []
        if not self.volume:
            tabs = [_running(t) for t in self.lines(x)]
        else:
            tabs = [t.transpose(1, 2).contiguous() for t in self.lines(x)]   # (B, L, S, N)
        for v in range(self.c["views"]):
            d = self.view(v)
            tab = tabs[0 if d["xb"] else 1]
            q = (d["d"] - d["p0"][:, None]) / d["pitch"][:, None]            # (L, n + 1)
            if not self.volume:
                o = (_at(tab, q).diff(dim=-1) * d["pitch"][:, None]).sum(1) * d["scale"]
            else:
                o = 0
                for l0 in range(0, tab.shape[1], 64):
                    ls = slice(l0, l0 + 64)
                    cols = _at(_running(tab[:, ls]), q[ls, None, :]).diff(dim=-1) * d["pitch"][ls, None, None]
                    zt = _running(cols, 2).transpose(2, 3)                    # (B, l, C, S + 1)
                    qz = (d["z"] - d["z0"][ls, None, None]) / d["zpitch"][ls, None, None]
                    o = o + (_at(zt, qz).diff(dim=-1) * d["zpitch"][ls, None, None]).sum(1)
                o = o.transpose(1, 2) * d["scale"]
            out.append(o.flip(-1) if d["flip"] else o)
        return torch.stack(out, 1)[:, None]

    def adjoint(self, y, weighted=False):
        y = y.double()[:, 0]
        b = y.shape[0]
        if not self.volume:
            acc = [torch.zeros((b, self.h, self.w), dtype=torch.float64, device=DEV),
                   torch.zeros((b, self.w, self.h), dtype=torch.float64, device=DEV)]
        else:
            acc = [torch.zeros((b, self.h, self.depth, self.w), dtype=torch.float64, device=DEV),
                   torch.zeros((b, self.w, self.depth, self.h), dtype=torch.float64, device=DEV)]
        for v in range(self.c["views"]):
            d = self.view(v)
            g = y[:, v].flip(-1) if d["flip"] else y[:, v]
            if not weighted:
                g = g * d["scale"]
            bnd = d["p0"][:, None] + d["pitch"][:, None] * torch.arange(d["npix"] + 1, dtype=torch.float64, device=DEV)
            k = (torch.searchsorted(d["d"], bnd.contiguous(), right=True) - 1).clamp(0, self.n - 1)
            w = d["d"].diff()
            q = k + ((bnd - d["d"][k]) / w[k]).clamp(0, 1)                    # (L, N + 1)
            fac = 1.0
            if weighted:
                cell = self.det if self.scan == "para" else d["cell"]
                fac = (cell / d["pitch"])[:, None]
                if self.volume:
                    fac = fac / d["zpitch"][:, None]
                if self.scan != "para":
                    ctr = ((torch.arange(d["npix"], dtype=torch.float64, device=DEV) + 0.5 - d["npix"] / 2)
                           * (self.sx if d["xb"] else self.sy) + (self.px if d["xb"] else self.py))[None, :]
                    xx, yy = (ctr, d["line"][:, None]) if d["xb"] else (d["line"][:, None], ctr)
                    sx, sy = d["srcxy"]
                    if self.fan_arc:
                        fac = fac / ((sx - xx) ** 2 + (sy - yy) ** 2)
                    else:
                        fac = fac * (self.iso / (self.iso - (sx * xx + sy * yy) / self.iso)) ** 2
            if not self.volume:
                acc[0 if d["xb"] else 1] += _at(_running(g * w)[:, None].expand(-1, q.shape[0], -1), q).diff(dim=-1) * fac
                continue
            # rows first: each column's integral over the rows at the slices' boundaries
            zr = d["z"]                                                       # (C, R + 1)
            seen = d["z0"][:, None] + d["zpitch"][:, None] * torch.arange(self.depth + 1, dtype=torch.float64,
                                                                           device=DEV)   # (L, S + 1)
            rt = _running(g, 1).transpose(1, 2)                               # (B, C, R + 1), per unit of row
            pitch = zr[:, 1] - zr[:, 0]
            dst = acc[0 if d["xb"] else 1]
            for l0 in range(0, dst.shape[1], 64):
                ls = slice(l0, l0 + 64)
                qz = (seen[ls, None, :] - zr[None, :, :1]) / pitch[None, :, None]       # (l, C, S + 1)
                n = qz.shape[0]
                a = _at(rt[:, None].expand(-1, n, -1, -1), qz).diff(dim=-1) * pitch[None, :, None]
                xt = _running((a * w[None, None, :, None]).transpose(2, 3))    # (B, l, S, C + 1)
                f = fac[ls, None, :] if weighted else 1.0
                dst[:, ls] += _at(xt, q[ls, None, :]).diff(dim=-1) * f
        if self.volume:
            acc = [t.transpose(1, 2) for t in acc]
        return (acc[0] + acc[1].transpose(-1, -2).flip(-2))[:, None]

    def fbp(self, y):
        n = self.n
        pitch = self.det if self.scan in ("para", "arc", "cone_arc", "spiral") else self.det * self.iso / self.sdd
        u = (torch.arange(n, dtype=torch.float64, device=DEV) - n / 2 + 0.5) * self.det + self.bins
        if not self.volume:
            wt = (torch.ones_like(u) if self.scan == "para" else torch.cos(u) if self.fan_arc else
                  self.iso / torch.sqrt((u * self.iso / self.sdd) ** 2 + self.iso ** 2))
        else:
            r = ((torch.arange(self.rows, dtype=torch.float64, device=DEV) - self.rows / 2 + 0.5) * self.drow
                 + self.rshift) * self.iso / self.sdd
            uc = torch.tan(u) * self.iso if self.fan_arc else u * self.iso / self.sdd
            wt = self.iso / torch.sqrt(r[:, None] ** 2 + uc[None] ** 2 + self.iso ** 2)
        i = torch.arange(n, device=DEV)
        off = (i[:, None] - i[None, :]).double()
        ramp = torch.where(off % 2 != 0, -1 / (math.pi * pitch * torch.where(off == 0, 1.0, off)) ** 2, 0.0)
        ramp = torch.where(off == 0, 1 / (4 * pitch * pitch), ramp)
        f = (y.double() * wt) @ ramp
        a = self.views.astype(np.float64)
        return self.adjoint(f, weighted=True) * (abs(a[-1] - a[0]) / (len(a) - 1) / 2)


def _scanner(case, g):
    return _Exact(case, g, _views(case, g), _table(case) if case["scan"] == "spiral" else None)


def exact(case, seed):
    with torch.no_grad():
        if case["scan"] == "uneven":
            xs, ys = _inputs(case, seed)
            g = _instance_geometry()
            parts = _instances(case)
            new = []
            for c, x, y in zip(parts, xs, ys):
                s = _scanner(c, g)
                new.append(x.double() - _ETA * s.adjoint(s.project(x) - y.double()))
            # slices of one scanner lie together, in order of their first appearance
            seen = {}
            for i, c in enumerate(parts):
                seen.setdefault((c["w"], c["dets"], c["views"]), []).append(i)
            return torch.cat([new[i].reshape(-1) for m in seen.values() for i in m])
        d = _inputs(case, seed)
        s = _scanner(case, _geometry(case))
        op = case["op"]
        if op == "project":
            return s.project(d["x"])
        if op == "adjoint":
            return s.adjoint(d["y"])
        if op == "fbp":
            return s.fbp(d["y"])
        p = s.project(d["x"])
        if op == "step":
            return [p, 2 * s.adjoint(p - d["y"].double())]
        back = s.fbp(p - d["y"].double())
        through = s.fbp(s.project(d["g"]))
        return [d["x"].double() - _WEIGHT * back, d["g"].double() - _WEIGHT * through, -(d["g"].double() * back).sum()]
