"""The work that a localisation program has this library do, as measurable cases.

A case is one call (or one short sequence of calls) of the package's public
entry points on inputs that such a program holds:

  device    fit_device: ROIs that lie in HBM, one model and box
  mixed     fit_mixed_device: groups of several models and boxes in one submission
  serve     Server: requests in pinned host memory, submitted together and waited for
  host      fit: numpy arrays in, a LocalizationResult with p-values out
  frames    cut_rois, fit_device and gmle_pvalues_device: resident frames to p-values
  generate  simulate_rois: synthetic ROI stacks on the device

Emitters have 500..5000 photons (astigmatic: 1500..15000, z between and just
around the two focal planes at +-50), 1..20 background photons per pixel, and
lie within 1.5 pixels of the ROI's centre, the distributions of the library's
synthetic workloads; sCMOS maps have lognormal read-noise variances (median
2 e-^2), gains of 0.4..0.6 e-/ADU and an offset of 100 ADU.
"""
from __future__ import annotations

import ctypes as C
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "gaussmle.jl_gb300"))

import gaussmle_gb300 as G  # noqa: E402
from gaussmle_gb300 import _lib, roofline, serve  # noqa: E402
from gaussmle_gb300.camera import ROIBatch, SCMOSCamera  # noqa: E402
from gaussmle_gb300.constraints import ParameterConstraints, default_constraints  # noqa: E402
from gaussmle_gb300.fitter import make_desc  # noqa: E402
from gaussmle_gb300.models import (AstigmaticXYZNB, GaussianXYNB, GaussianXYNBS,  # noqa: E402
                                   GaussianXYNBSXSY)

ITERATIONS = 20
NPAR = {0: 4, 1: 5, 2: 6, 3: 5}
# fractions, models and boxes of the mixed sCMOS batch
MIX = [(0.40, 0, 11), (0.25, 1, 9), (0.15, 2, 13), (0.15, 3, 15), (0.05, 0, 7)]
CELL = 16  # frames: one emitter per cell of this many pixels, boxes up to 15


def listed():
    return [
        # one camera frame of a live acquisition: latency and launch cost
        {"name": "frame-xynb11-200", "path": "device", "model": 0, "box": 11, "camera": 0, "n": 200},
        # the fitter's default batch size
        {"name": "batch-xynb11-10k", "path": "device", "model": 0, "box": 11, "camera": 0,
         "n": 10_000},
        # a whole acquisition, ideal camera: the headline box and model
        {"name": "batch-xynb11-1m", "path": "device", "model": 0, "box": 11, "camera": 0,
         "n": 1_000_000},
        # a whole acquisition of raw sCMOS counts with a fitted width
        {"name": "batch-xynbs13-scmos-1m", "path": "device", "model": 1, "box": 13, "camera": 2,
         "n": 1_000_000},
        # even box, odd count, data already in electrons, two fitted widths
        {"name": "batch-xynbsxsy10-var-100k", "path": "device", "model": 2, "box": 10, "camera": 1,
         "n": 99_991},
        # a 3-D acquisition, ideal camera
        {"name": "batch-astig15-300k", "path": "device", "model": 3, "box": 15, "camera": 0,
         "n": 300_000},
        # 3-D with a wide point spread: ROIs beyond 16 pixels
        {"name": "batch-astig21-scmos-12k", "path": "device", "model": 3, "box": 21, "camera": 2,
         "n": 12_000},
        # the mixed sCMOS batch: large and small groups of five kinds in one submission
        {"name": "mixed-scmos-500k", "path": "mixed", "camera": 2, "n": 500_000, "groups": 5},
        # requests of many sizes from pinned host memory through the serving loop
        {"name": "serve-scmos-100k", "path": "serve", "camera": 2, "n": 100_000, "groups": 40},
        # the ordinary Python call on numpy arrays
        {"name": "call-xynb11-scmos-50k", "path": "host", "model": 0, "box": 11, "camera": 2,
         "n": 50_000},
        # frames on the GPU to localisations with goodness of fit
        {"name": "frames-xynbs9-scmos-200k", "path": "frames", "model": 1, "box": 9, "camera": 2,
         "n": 200_000},
        # synthetic sCMOS stacks for validation runs
        {"name": "generate-xynb11-scmos-200k", "path": "generate", "model": 0, "box": 11,
         "camera": 2, "n": 200_000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choices(["device", "mixed", "serve", "host", "frames", "generate"],
                       [45, 11, 11, 11, 11, 11])[0]
    if path in ("mixed", "serve"):
        n = _log_int(rng, 2_000, 500_000 if path == "mixed" else 100_000)
        return {"path": path, "camera": rng.choice([0, 1, 2]), "n": n,
                "groups": rng.randint(5, 60)}
    model, camera = rng.randrange(4), rng.choice([0, 1, 2])
    if path == "host" and camera == 1:
        camera = 2  # an SCMOSCamera's batches are in ADU
    lo = {0: 5, 1: 7, 2: 9, 3: 13}[model]
    box = rng.randint(lo, 16 if path == "device" else 15)
    top = {"device": 300_000, "host": 100_000, "frames": 200_000, "generate": 300_000}[path]
    if path == "device" and rng.random() < 0.25:
        box, top = rng.randint(17, 32), 12_000
    top = int(top * min(1.0, (13.0 if box <= 16 else 21.0) ** 2 / box ** 2))
    return {"path": path, "model": model, "box": box, "camera": camera, "n": _log_int(rng, 64, top)}


# ---- inputs --------------------------------------------------------------------

def _psf(model):
    if model == 3:
        return AstigmaticXYZNB(1.3, 1.3, 0.05, 0.05, 0.3, 0.3, 50.0, 100.0)
    return {0: GaussianXYNB(1.3), 1: GaussianXYNBS(), 2: GaussianXYNBSXSY()}[model]


def _constraints(model, box):
    if model == 3:
        return ParameterConstraints([-2, -2, -600, 1, 0.01], [box + 2, box + 2, 600, np.inf, np.inf],
                                    [1, 1, 60, 100, 2])
    return default_constraints(_psf(model), box)


def _sensor(case):
    return 2048 if case["n"] >= 100_000 and case["path"] in ("device", "mixed") else 512


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _maps(g, sensor):
    """(variance, gain, offset) as (nx, ny) tensors: Julia's column-major (ny, nx)."""
    kw = dict(generator=g, device=_dev())
    var = torch.exp(math.log(2.0) + 0.5 * torch.randn((sensor, sensor), **kw))
    gain = 0.4 + 0.2 * torch.rand((sensor, sensor), **kw)
    return var, gain, torch.full((sensor, sensor), 100.0, device=_dev())


def _truth(g, model, box, n):
    u = lambda a, b: a + (b - a) * torch.rand(n, generator=g, device=_dev(), dtype=torch.float64)
    c = (box + 1) / 2.0
    x, y, bg = u(c - 1.5, c + 1.5), u(c - 1.5, c + 1.5), u(1, 20)
    if model == 3:
        cols = [x, y, u(-80, 80), u(1500, 15000), bg]
    else:
        cols = [x, y, u(500, 5000), bg]
        cols += [u(1.0, 1.8)] if model == 1 else [u(1.0, 1.9), u(1.0, 1.9)] if model == 2 else []
    return torch.stack(cols, 1).float()


def _widths(model, th, psf):
    """sigma_x, sigma_y of parameter rows th, and for the astigmatic model the
    first and second derivatives of both with respect to z."""
    if model == 0:
        s = torch.full_like(th[:, 0], float(np.float32(psf[0])))
        return s, s, None
    if model == 1:
        return th[:, 4], th[:, 4], None
    if model == 2:
        return th[:, 4], th[:, 5], None
    out, der = [], []
    sx0, sy0, Ax, Ay, Bx, By, gamma, d = (float(np.float32(v)) for v in psf)
    for s0, A, B, zz in ((sx0, Ax, Bx, th[:, 2] - gamma), (sy0, Ay, By, th[:, 2] + gamma)):
        q = zz / d
        a = 1 + q ** 2 + A * q ** 3 + B * q ** 4
        da = (2 * q + 3 * A * q ** 2 + 4 * B * q ** 3) / d
        dda = (2 + 6 * A * q + 12 * B * q ** 2) / d ** 2
        out.append(s0 * a.sqrt())
        der += [s0 / (2 * a.sqrt()) * da, s0 / (2 * a.sqrt()) * dda - s0 / (4 * a ** 1.5) * da ** 2]
    return out[0], out[1], der


def _edges(c, s, box):
    """Offsets of the pixel edges from the centre, erf and Gaussian at them: (n, box + 1)."""
    u = torch.arange(box + 1, device=c.device, dtype=c.dtype)[None] + 0.5 - c[:, None]
    t = u / s[:, None]
    return u, torch.erf(t * math.sqrt(0.5)), torch.exp(-0.5 * t * t)


def _mu(model, th, psf, box):
    """Expected photons (n, box, box): [ROI, column, row]."""
    th = th.double()
    sx, sy, _ = _widths(model, th, psf)
    px, py = (0.5 * e.diff(dim=1) for e in (_edges(th[:, 0], sx, box)[1], _edges(th[:, 1], sy, box)[1]))
    iN, ib = (3, 4) if model == 3 else (2, 3)
    return th[:, ib, None, None] + th[:, iN, None, None] * px[:, :, None] * py[:, None, :]


def _tiles(m, xc, yc, box):
    k = torch.arange(box, device=m.device)
    return m[(xc.long() - 1)[:, None, None] + k[None, :, None],
             (yc.long() - 1)[:, None, None] + k[None, None, :]]


def _rois(g, model, box, camera, n, maps, xc=None, yc=None):
    """ROIs of `n` emitters: (data (n, box, box), xc, yc)."""
    kw = dict(generator=g, device=_dev())
    th = _truth(g, model, box, n)
    if camera and xc is None:
        side = maps[0].shape[0]
        xc = torch.randint(1, side - box + 2, (n,), dtype=torch.int32, **kw)
        yc = torch.randint(1, side - box + 2, (n,), dtype=torch.int32, **kw)
    data = torch.empty((n, box, box), device=_dev())
    psf, step = _psf(model).psf_vector(), 1 << 17
    for k in range(0, n, step):
        part = slice(k, min(n, k + step))
        e = torch.poisson(_mu(model, th[part], psf, box).float().clamp_(min=0), generator=g)
        if camera:
            v, gn, off = (_tiles(m, xc[part], yc[part], box) for m in maps)
            e += torch.randn(e.shape, **kw) * v.sqrt()
            if camera == 2:
                e = e / gn + off
        data[part] = e
    return data, xc, yc


def _group_sizes(rng, n, groups):
    """(model, box, count) of a mixed submission: the MIX proportions of n ROIs, in about
    `groups` groups of unequal sizes."""
    out = []
    for f, model, box in MIX:
        left, parts = max(1, int(f * n)), max(1, round(f * groups))
        cuts = sorted(int(left * rng.random()) for _ in range(parts - 1))
        out += [(model, box, b - a) for a, b in zip([0] + cuts, cuts + [left]) if b > a]
    return out


def _context(maps=None):
    ctx = _lib.Context(0)
    if maps is not None:
        var, gain, off = (np.ascontiguousarray(m.cpu().numpy()) for m in maps)
        p = lambda a: a.ctypes.data_as(C.c_void_p)
        ctx.check(ctx.lib.gmle_set_calibration(ctx.handle, p(var), p(gain), p(off),
                                               var.shape[1], var.shape[0]))
    return ctx


def _outputs(n, P, **kw):
    return {"params": torch.empty((n, P), **kw), "crlb": torch.empty((n, P), **kw),
            "llr": torch.empty(n, **kw), "flags": torch.empty(n, dtype=torch.uint8, **kw)}


def _inputs(case, seed):
    """Everything of a case that does not need the library: plain tensors."""
    g = torch.Generator(device=_dev())
    g.manual_seed(seed)
    path, camera, n = case["path"], case["camera"], case["n"]
    maps = _maps(g, _sensor(case)) if camera else None
    if path in ("mixed", "serve"):
        sizes = _group_sizes(np.random.default_rng(n + case["groups"]), n, case["groups"])
        return {"maps": maps, "parts": [(m, b, *_rois(g, m, b, camera, k, maps))
                                        for m, b, k in sizes]}
    model, box = case["model"], case["box"]
    if path == "generate":
        xc = yc = None
        if camera:
            xc, yc = (torch.randint(1, maps[0].shape[0] - box + 2, (n,), generator=g,
                                    device=_dev(), dtype=torch.int32) for _ in range(2))
        return {"maps": maps, "truth": _truth(g, model, box, n), "xc": xc, "yc": yc}
    if path == "frames":
        side, cells = 512, (512 // CELL) ** 2
        frames = max(1, -(-n // (cells // 2)))  # about half of the cells hold an emitter
        at = torch.randperm(frames * cells, generator=g, device=_dev())[:n].sort().values
        fidx, cell = (at // cells).int() + 1, at % cells
        corner = lambda c: (c * CELL + torch.randint(1, CELL - box + 2, (n,), generator=g,
                                                     device=_dev())).int()
        xc, yc = corner(cell // (512 // CELL)), corner(cell % (512 // CELL))
        rois, _, _ = _rois(g, model, box, camera, n, maps, xc, yc)
        stack = torch.poisson(torch.full((frames, side, side), 10.0, device=_dev()), generator=g)
        if camera == 2:
            stack = stack / maps[1] + maps[2]
        k = torch.arange(box, device=_dev())
        stack[(fidx.long() - 1)[:, None, None], (xc.long() - 1)[:, None, None] + k[None, :, None],
              (yc.long() - 1)[:, None, None] + k[None, None, :]] = rois
        return {"maps": maps, "frames": stack, "fidx": fidx, "xc": xc, "yc": yc, "rois": rois}
    rois, xc, yc = _rois(g, model, box, camera, n, maps)
    return {"maps": maps, "rois": rois, "xc": xc, "yc": yc}


def prepare(case, seed):
    w = _inputs(case, seed)
    path, camera = case["path"], case["camera"]
    s = {"path": path, "case": case, "ctx": _context(w["maps"])}
    if path in ("mixed", "serve"):
        s["groups"], s["out"], s["keep"] = [], [], []
        kw = {"device": _dev()} if path == "mixed" else {"pin_memory": True}
        for m, b in dict.fromkeys(p[:2] for p in w["parts"]):
            # the results of one model and box lie in one set of arrays
            parts = [p[2:] for p in w["parts"] if p[:2] == (m, b)]
            o, at = _outputs(sum(p[0].shape[0] for p in parts), NPAR[m], **kw), 0
            for rois, xc, yc in parts:
                if path == "serve":
                    rois, xc, yc = (None if t is None else t.cpu().pin_memory()
                                    for t in (rois, xc, yc))
                to = slice(at, at + rois.shape[0])
                at = to.stop
                s["groups"].append(serve.make_group(
                    _psf(m), b, camera, _constraints(m, b), rois, xc, yc,
                    *(o[k][to] for k in ("params", "crlb", "llr", "flags"))))
                s["keep"].append((rois, xc, yc))
            s["out"].append(o)
        if path == "serve":
            s["server"] = serve.Server(s["ctx"], hbm_budget_bytes=256 << 20)
            s["requests"] = (_lib.Group * len(s["groups"]))(*s["groups"])
        return s
    model, box, n = case["model"], case["box"], case["n"]
    if path == "host":
        data = np.asfortranarray(w["rois"].cpu().numpy().transpose(2, 1, 0))
        psf = GaussianXYNB(0.13) if model == 0 else \
            AstigmaticXYZNB(0.13, 0.13, 0.05, 0.05, 0.3, 0.3, 50.0, 100.0) if model == 3 else _psf(model)
        s["fitter"] = G.GaussMLEFitter(psf_model=psf, context=s["ctx"],
                                       constraints=_constraints(model, box))
        s["data"] = data
        if camera:
            var, gain, off = (m.cpu().numpy().T for m in w["maps"])
            cam = SCMOSCamera(var.shape[1], var.shape[0], 0.1, np.sqrt(var), off, gain)
            s["data"] = ROIBatch(data, w["xc"].cpu().numpy(), w["yc"].cpu().numpy(),
                                 np.ones(n, np.int32), cam)
        return s
    s["desc"] = make_desc(_psf(model), box, ITERATIONS, _constraints(model, box), camera)
    s["xc"], s["yc"] = w["xc"], w["yc"]
    if path == "generate":
        s.update(truth=w["truth"], seed=seed, out=torch.empty(n * box * box, device=_dev()))
        return s
    s["out"] = _outputs(n, NPAR[model], device=_dev())
    if path == "frames":
        s.update(frames=w["frames"], fidx=w["fidx"], rois=torch.empty(n * box * box, device=_dev()))
        s["out"]["pvalues"] = torch.empty(n, device=_dev())
    else:
        s["rois"] = w["rois"]
    return s


# ---- one pass -------------------------------------------------------------------

def run(s):
    path, ctx, case = s["path"], s["ctx"], s["case"]
    if path == "mixed":
        serve.fit_mixed_device(ctx, s["groups"])
        return s["out"]
    if path == "serve":
        for t in s["server"].submit_many(s["requests"]):
            s["server"].wait(t)
        return s["out"]
    if path == "host":
        r = G.fit(s["fitter"], s["data"])
        return {"params": r.params, "crlb": r.uncertainties, "llr": r.log_likelihoods,
                "flags": r.flags, "pvalues": r.pvalues, "x": r.x_camera, "y": r.y_camera}
    if path == "generate":
        G.simulate_rois(ctx, s["desc"], s["truth"], s["seed"], s["xc"], s["yc"], out=s["out"])
        return s["out"]
    o = s["out"]
    if path == "frames":
        G.cut_rois(ctx, s["frames"], s["fidx"], s["xc"], s["yc"], case["box"], out=s["rois"])
    G.fit_device(ctx, s["desc"], s["rois"], s["xc"], s["yc"], o["params"], o["crlb"], o["llr"],
                 o["flags"])
    if path == "frames":
        p = lambda t: C.c_void_p(t.data_ptr())
        ctx.check(ctx.lib.gmle_pvalues_device(
            ctx.handle, p(o["llr"]), case["n"], case["box"] ** 2 - NPAR[case["model"]],
            p(o["pvalues"]), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return o


def work(case):
    path, camera, n = case["path"], case["camera"], case["n"]

    def fits(model, box, k):
        w = roofline.work_per_roi(model, box, ITERATIONS, camera)
        return k * (w["fp32"] + w["sfu"]), k * roofline.bytes_per_roi(model, box, camera)

    if path in ("mixed", "serve"):
        parts = [fits(m, b, f * n) for f, m, b in MIX]
        return {"flops": sum(p[0] for p in parts), "bytes": sum(p[1] for p in parts)}
    model, box = case["model"], case["box"]
    if path == "generate":
        # ten Philox rounds, the sampler's arithmetic and the noise of each pixel
        maps = {0: 0, 1: 4, 2: 12}[camera]
        return {"flops": 100.0 * n * box * box,
                "bytes": n * (box * box * (4 + maps) + 4 * NPAR[model] + 8)}
    flops, size = fits(model, box, n)
    # frames: the ROIs' pixels come straight from the frames; p-values go out
    return {"flops": flops, "bytes": size + (8 * n if path == "frames" else 4 * n if path == "host"
                                             else 0)}


# ---- the same fits in 64 bits ------------------------------------------------------

def _derivatives(c, s, N, box, sigma):
    """Along one axis: psf and, without the other axis' psf, d and d2 with respect to the
    position and (sigma) to the width."""
    u, erf, gau = _edges(c, s, box)
    k = (-N / math.sqrt(2 * math.pi) / s)[:, None]
    s = s[:, None]
    ug = u * gau
    out = [0.5 * erf.diff(dim=1), k * gau.diff(dim=1), k / s ** 2 * ug.diff(dim=1)]
    if sigma:
        d1 = k / s * ug.diff(dim=1)
        out += [d1, -2 / s * d1 + k / s ** 4 * (u ** 3 * gau).diff(dim=1)]
    return out


def _model(model, th, psf, box):
    """mu, and per parameter the first and second derivative as lists of (column factor,
    row factor) products, each (n, box)."""
    iN, ib = (3, 4) if model == 3 else (2, 3)
    sx, sy, dz = _widths(model, th, psf)
    x = _derivatives(th[:, 0], sx, th[:, iN], box, model > 0)
    y = _derivatives(th[:, 1], sy, th[:, iN], box, model > 0)
    one, zero = torch.ones_like(x[0]), torch.zeros_like(x[0])
    d1 = {0: [(x[1], y[0])], 1: [(x[0], y[1])], iN: [(x[0], y[0])], ib: [(one, one)]}
    d2 = {0: [(x[2], y[0])], 1: [(x[0], y[2])], iN: [(zero, zero)], ib: [(zero, zero)]}
    if model == 1:
        d1[4] = [(x[3], y[0]), (x[0], y[3])]
        d2[4] = [(x[4], y[0]), (x[0], y[4])]
    elif model == 2:
        d1[4], d2[4] = [(x[3], y[0])], [(x[4], y[0])]
        d1[5], d2[5] = [(x[0], y[3])], [(x[0], y[4])]
    elif model == 3:
        ax, aax, ay, aay = (v[:, None] for v in dz)
        d1[2] = [(x[3] * ax, y[0]), (x[0], y[3] * ay)]
        d2[2] = [(x[4] * ax ** 2 + x[3] * aax, y[0]), (x[0], y[4] * ay ** 2 + y[3] * aay)]
    mu = th[:, ib, None, None] + th[:, iN, None, None] * x[0][:, :, None] * y[0][:, None, :]
    full = lambda t: sum(a[:, :, None] * b[:, None, :] for a, b in t)
    return mu, (lambda k: full(d1[k])), (lambda k: full(d2[k]))


def _start(model, box, d, psf):
    n = d.shape[0]
    rim = torch.ones((box, box), dtype=torch.bool, device=d.device)
    rim[1:-1, 1:-1] = False
    bg = d[:, rim].mean(1)
    sig = (d - bg[:, None, None]).clamp(min=0)
    total = sig.sum((1, 2))
    t = torch.arange(1, box + 1, device=d.device, dtype=d.dtype)
    sx, sy = sig.sum(2), sig.sum(1)
    centre = torch.full_like(total, (box + 1) / 2.0)
    x, y = (torch.where(total > 10, (s * t).sum(1) / total, centre).clamp(1.5, box - 0.5)
            for s in (sx, sy))
    cols = [x, y, total.clamp(min=100), bg]
    if model in (1, 2):
        cols += [torch.full_like(x, float(np.float32(1.3)))] * model
    if model == 3:
        wx, wy = (((s * (t[None] - c[:, None]) ** 2).sum(1) / total).clamp(min=0.5)
                  for s, c in ((sx, x), (sy, y)))
        z = -(wx / float(psf[0]) ** 2 - wy / float(psf[1]) ** 2) * float(psf[7]) ** 2 / (4 * float(psf[6]))
        cols.insert(2, torch.where(total > 10, z.clamp(-600, 600), torch.zeros_like(z)))
    return torch.stack(cols, 1).reshape(n, -1)


def _fit64(model, box, camera, rois, maps, xc, yc, psf=None, cons=None):
    """params, crlb and llr of the ROIs by the library's iteration, in 64 bits."""
    psf = np.float32(_psf(model).psf_vector() if psf is None else psf)
    cons = _constraints(model, box) if cons is None else cons
    lo, hi, most = (torch.from_numpy(np.asarray(v, np.float64)).to(rois.device)
                    for v in (cons.lower, cons.upper, cons.max_step))
    P, outs = NPAR[model], []
    for k in range(0, rois.shape[0], 1 << 16):
        d = rois[k:k + (1 << 16)].double()
        v = 0.0
        if camera:
            part = (xc[k:k + (1 << 16)], yc[k:k + (1 << 16)], box)
            v = _tiles(maps[0], *part).double()
            if camera == 2:
                d = (d - _tiles(maps[2], *part).double()) * _tiles(maps[1], *part).double()
        th = _start(model, box, d, psf)
        for _ in range(ITERATIONS):
            mu, d1, d2 = _model(model, th, psf, box)
            if camera:
                cf, df = (d - mu) / (mu + v), 1 / (mu + v)
            else:
                pos = mu > float(np.float32(0.01))
                cf = torch.where(pos, (d / mu - 1).clamp(max=1e4), torch.zeros_like(mu))
                df = torch.where(pos, (d / mu ** 2).clamp(max=1e4), torch.zeros_like(mu))
            new = []
            for p in range(P):
                a = d1(p)
                grad, hess = (a * cf).sum((1, 2)), (d2(p) * cf - a * a * df).sum((1, 2))
                step = torch.where(hess.abs() > 1e-10, grad / hess, torch.zeros_like(grad))
                new.append((th[:, p] - step.clamp(-most[p], most[p])).clamp(lo[p], hi[p]))
            th = torch.stack(new, 1)
        mu, d1, _ = _model(model, th, psf, box)
        a = torch.stack([d1(p) for p in range(P)], 1).flatten(2)
        w = torch.where(mu > 0, 1 / (mu + v), torch.zeros_like(mu)).flatten(1)
        F = torch.einsum("npk,nqk,nk->npq", a, a, w)
        F = F + 1e-10 * F.abs().amax((1, 2))[:, None, None] * torch.eye(P, device=F.device,
                                                                       dtype=F.dtype)
        crlb = torch.linalg.inv(F).diagonal(dim1=1, dim2=2).clamp(min=0).sqrt()
        if camera:
            llr = (-0.5 * (d - mu) ** 2 / (mu + v)).sum((1, 2))
        else:
            llr = (torch.xlogy(d, mu) - mu - torch.xlogy(d, d) + d).sum((1, 2))
        outs.append((th, crlb, llr))
    return tuple(torch.cat(t) for t in zip(*outs))


def _pvalues64(llr, df):
    """1 - P(df / 2, -llr): the chance of a chi-square of df degrees above -2 llr."""
    x = (-llr).clamp(min=0)
    return 1 - torch.special.gammainc(torch.full_like(x, df / 2.0), x)


def exact(case, seed):
    path, camera = case["path"], case["camera"]
    if path == "generate":
        return None  # draws of the generator's own random streams
    w = _inputs(case, seed)

    def row(r):
        return {"params": r[0], "crlb": r[1], "llr": r[2], "flags": None}

    if path in ("mixed", "serve"):
        kinds = {}
        for m, b, rois, xc, yc in w["parts"]:
            kinds.setdefault((m, b), []).append(_fit64(m, b, camera, rois, w["maps"], xc, yc))
        return [row([torch.cat(t) for t in zip(*fits)]) for fits in kinds.values()]
    model, box = case["model"], case["box"]
    psf = _psf(model).psf_vector()
    maps = w["maps"]
    if path == "host":
        if model in (0, 3):  # given in microns, 0.1 micron pixels
            scale = np.float32(0.13) / np.float32(0.1)
            psf[:1 if model == 0 else 2] = scale
        if camera:  # the camera holds the read noise, its square is the variance
            rn = maps[0].sqrt()
            maps = (rn * rn, maps[1], maps[2])
    th, crlb, llr = _fit64(model, box, camera, w["rois"], maps, w["xc"], w["yc"], psf)
    out = row((th, crlb, llr))
    if path in ("host", "frames"):
        out["pvalues"] = _pvalues64(llr, box * box - NPAR[model])
    if path == "host":
        n = th.shape[0]
        xc = w["xc"] if camera else 1 + box * torch.arange(n, device=th.device)
        yc = w["yc"] if camera else torch.ones(n, device=th.device)
        out["x"], out["y"] = xc.double() + th[:, 0] - 1, yc.double() + th[:, 1] - 1
    return out
