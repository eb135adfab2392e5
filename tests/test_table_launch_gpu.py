"""Table launches of sCMOS groups in the shapes that submissions take by default: a
warp per ROI, and 16x16 boxes in blocks of 224 ROIs, one block per tile
(gmle_fit_mixed_device) and persistent, with more tiles than resident blocks, so that
a block takes its tensor memory for several tiles (gmle_fit_mixed_device_noalloc).
A ROI's bits are those of the plain launch in the same kernel."""
import ctypes as C

import numpy as np
import pytest

import gaussmle_gb300 as G
from gaussmle_gb300 import _lib, serve
from gaussmle_gb300.fitter import make_desc
from parity_cases import make_case
from test_edge_gpu import set_maps

pytestmark = pytest.mark.gpu


def device_batch(w, repeat=1, n=None):
    """The workload's ROIs over and over, up to n, on the device: data, xc, yc."""
    torch = pytest.importorskip("torch")
    b2 = w.box * w.box
    n = n or w.n
    data = torch.from_numpy(np.ascontiguousarray(w.data.transpose(2, 1, 0)).reshape(-1, b2)).cuda()
    xc, yc = torch.from_numpy(w.x_corners).cuda(), torch.from_numpy(w.y_corners).cuda()
    return [t.repeat(*([repeat] + [1] * (t.dim() - 1)))[:n].contiguous() for t in (data, xc, yc)]


def outputs(n, P):
    torch = pytest.importorskip("torch")
    f = dict(dtype=torch.float32, device="cuda")
    return [torch.full((n, P), 7.0, **f), torch.full((n, P), 7.0, **f), torch.full((n,), 7.0, **f),
            torch.zeros(n, dtype=torch.uint8, device="cuda")]


def plain(ctx, w, batch, out):
    import torch
    G.fit_device(ctx, make_desc(w.psf, w.box, 20, w.constraints, w.camera), batch[0].reshape(-1),
                 batch[1], batch[2], *out)
    torch.cuda.synchronize()


def same(a, b):
    for x, y in zip(a, b):
        assert np.array_equal(x.cpu().numpy(), y.cpu().numpy(), equal_nan=True)


@pytest.mark.parametrize("camera", [1, 2])
def test_a_warp_per_roi_from_a_table(ctx, camera):
    import torch
    # 2 x 1475 ROIs, below 20 per SM (152 SMs)
    ws = [make_case(f"m{m}-{b}-{camera}", m, b, camera, n, seed=90 + b)
          for m, b, n in [(0, 4, 1), (0, 11, 600), (1, 16, 33), (2, 9, 301), (1, 13, 450), (3, 15, 90)]]
    set_maps(ctx, ws[0].maps)
    batches = [device_batch(w) for w in ws] * 2  # two groups of each kind
    outs = [outputs(w.n, w.psf.nparams) for w in ws + ws]
    serve.fit_mixed_device(ctx, [
        serve.make_group(w.psf, w.box, camera, w.constraints, b[0].reshape(-1), b[1], b[2], *o)
        for w, b, o in zip(ws + ws, batches, outs)])
    torch.cuda.synchronize()
    for w, b, o in zip(ws + ws, batches, outs):
        want = outputs(w.n, w.psf.nparams)
        plain(ctx, w, b, want)
        same(o, want)


# n: the ROIs of each of two groups.  16x16, from 38 912 ROIs in all: blocks of 224, of
# which one is resident per SM, so 181 tiles for 152; 11x11: blocks of 128, 574 tiles.
@pytest.mark.parametrize("model,box,n", [(0, 16, 20_201), (3, 16, 20_201), (0, 11, 36_600)])
@pytest.mark.parametrize("persistent", [False, True])
def test_one_thread_per_roi_from_a_table(ctx, model, box, n, persistent):
    import torch
    w = make_case(f"m{model}-{box}-2", model, box, 2, 500)
    set_maps(ctx, w.maps)
    batch = device_batch(w, -(-2 * n // 500), 2 * n)
    got, want = outputs(2 * n, w.psf.nparams), outputs(2 * n, w.psf.nparams)
    ctx.check(ctx.lib.gmle_set_tuning(ctx.handle, model, box, 2, 1, 128))
    try:
        plain(ctx, w, batch, want)
    finally:
        ctx.check(ctx.lib.gmle_set_tuning(ctx.handle, model, box, 2, 0, 0))
    torch.cuda.synchronize()
    gs = [serve.make_group(w.psf, box, 2, w.constraints, batch[0][k].reshape(-1), batch[1][k],
                           batch[2][k], *(o[k] for o in got))
          for k in (slice(0, n - 57), slice(n - 57, 2 * n))]
    if persistent:
        maps = [torch.from_numpy(np.ascontiguousarray(m.T, np.float32)).cuda() for m in w.maps]
        err, (ny, nx) = C.create_string_buffer(512), w.maps[0].shape
        st = ctx.lib.gmle_fit_mixed_device_noalloc(
            (_lib.Group * 2)(*gs), 2, *(C.c_void_p(m.data_ptr()) for m in maps), ny, nx, None, err,
            512)
        assert st == 0, err.value
    else:
        serve.fit_mixed_device(ctx, gs)
    torch.cuda.synchronize()
    same(got, want)
