"""The kernels' corner check (csrc/gmle_corners.h), compiled for the host: corners
that leave the maps are outside for every int32, also where the corner plus the box
overflows."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from gaussmle_gb300 import build

I32 = 2 ** 31


@pytest.fixture(scope="module")
def inside(tmp_path_factory):
    d = tmp_path_factory.mktemp("corners")
    (d / "c.cpp").write_text('#include "gmle_corners.h"\nextern "C" int inside(int x, int y, int b, '
                             'int ny, int nx) { return gmle::corner_inside(x, y, b, ny, nx); }\n')
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", f"-I{build.CSRC}", str(d / "c.cpp"), "-o",
                    str(d / "c.so")], check=True)
    return C.CDLL(str(d / "c.so")).inside


@pytest.mark.parametrize("box", [3, 11, 16, 64])
@pytest.mark.parametrize("ny,nx", [(256, 300), (64, 64), (5, 5), (0, 0), (46_000, 46_000)])
def test_corner_inside(inside, box, ny, nx):
    edge = [-I32, -1, 0, 1, 2, I32 - 1, I32 - 2, I32 - box, I32 - box + 1, I32 - box + 2]
    xs = sorted({v for v in edge + [nx - box, nx - box + 1, nx - box + 2, nx] if v < I32})
    ys = sorted({v for v in edge + [ny - box, ny - box + 1, ny - box + 2, ny] if v < I32})
    for x in xs:
        for y in ys:
            want = x >= 1 and y >= 1 and x + box - 1 <= nx and y + box - 1 <= ny
            assert bool(inside(x, y, box, ny, nx)) == want, (x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("box,n,shape", [(11, 40, None), (15, 40, (4, 32)), (13, 40, (1, 32)),
                                         (11, 40, (1, 32)), (21, 40, None), (33, 9, None)])
def test_kernels_skip_and_count_corners_near_the_largest_int(ctx, box, n, shape):
    torch = pytest.importorskip("torch")
    import gaussmle_gb300 as G
    from gaussmle_gb300.fitter import make_desc
    from parity_cases import make_case
    from test_edge_gpu import set_maps
    w = make_case(f"m0-{box}-2", 0, box, 2, n)
    set_maps(ctx, w.maps)
    xc, yc = w.x_corners.copy(), w.y_corners.copy()
    xc[1], yc[2], xc[3] = I32 - 1, I32 - 1, I32 - box + 2
    xc[5] = yc[5] = I32 - 1
    bad = [1, 2, 3, 5]
    dev = torch.device("cuda", 0)
    out = [torch.empty((n, 4), device=dev), torch.empty((n, 4), device=dev),
           torch.empty(n, device=dev), torch.empty(n, dtype=torch.uint8, device=dev)]
    data = torch.from_numpy(np.ascontiguousarray(w.data.transpose(2, 1, 0)).reshape(-1)).to(dev)
    count = C.c_int64()
    ctx.check(ctx.lib.gmle_fit_device_errors(ctx.handle, C.byref(count)))
    if shape:
        ctx.check(ctx.lib.gmle_set_tuning(ctx.handle, 0, box, 2, *shape))
    try:
        G.fit_device(ctx, make_desc(w.psf, box, 20, w.constraints, 2), data,
                     torch.from_numpy(xc).to(dev), torch.from_numpy(yc).to(dev), *out)
        ctx.check(ctx.lib.gmle_fit_device_errors(ctx.handle, C.byref(count)))
    finally:
        if shape:
            ctx.check(ctx.lib.gmle_set_tuning(ctx.handle, 0, box, 2, 0, 0))
    assert count.value == len(bad)
    prm, flags = out[0].cpu().numpy(), out[3].cpu().numpy()
    assert np.isnan(prm[bad]).all() and np.isfinite(np.delete(prm, bad, 0)).all()
    assert not flags[bad].any()
