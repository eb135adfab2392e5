"""Small batches of boxes 3..16, fitted with one warp per ROI by default: the edges
of the lane grid (4, 8, 12, 15/16 pixels), blocks with empty warps, the table
launch of a mixed submission, and both sides of the line of 20 ROIs per SM.
Compared with the oracle at the parity bar (test_boxes_gpu.check); the start
point bit for bit (the sums run in the reference's order)."""
import numpy as np
import pytest

import gaussmle_gb300 as G
from gaussmle_gb300 import serve
from gaussmle_gb300.fitter import make_desc
from oracle import oracle as O
from parity_cases import make_case, oracle_desc
from test_boxes_gpu import check
from test_edge_gpu import host_fit, set_maps
from test_parity_gpu import run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,camera", [(0, 0), (1, 2), (2, 1), (3, 0)])
@pytest.mark.parametrize("box,n", [(5, 1), (7, 305), (8, 3), (9, 610), (12, 5), (13, 2), (15, 307),
                                   (16, 914)])
def test_lane_grid_edges(ctx, model, camera, box, n):
    if model and box < 7 or model == 3 and (box < 13 or n < 100):
        pytest.skip("too few pixels for the model, or too few ROIs for its pass rate")
    w = make_case(f"m{model}-{box}-{camera}", model, box, camera, n)
    params, crlb, llr, flags = run_gpu(ctx, w)
    check(w, params, crlb, flags)


@pytest.mark.parametrize("box", [3, 4, 8, 9, 12, 15, 16])
@pytest.mark.parametrize("model,camera", [(0, 0), (2, 2), (3, 1)])
def test_start_point_is_the_references(ctx, model, camera, box):
    w = make_case(f"m{model}-{box}-{camera}", model, box, camera, 50)
    if w.camera:
        set_maps(ctx, w.maps)
    desc = make_desc(w.psf, box, 0, w.constraints, camera)
    st, (prm, *_) = host_fit(ctx, desc, w.data, w.x_corners, w.y_corners)
    ctx.check(st)
    ref = O.fit(oracle_desc(O, w, iterations=0), w.data, w.x_corners, w.y_corners, w.maps)
    assert np.array_equal(prm, ref["params"])


@pytest.mark.parametrize("n", [3039, 3040, 3041])
def test_both_sides_of_the_line(ctx, n):
    w = make_case("xynb-11-poisson", 0, 11, 0, n)
    params, crlb, llr, flags = run_gpu(ctx, w)
    check(w, params, crlb, flags)


@pytest.mark.parametrize("model,box,camera,n", [(1, 5, 0, 4864), (1, 5, 0, 4865),
                                                (1, 9, 0, 9728), (1, 9, 0, 9729),
                                                (0, 11, 2, 14592), (0, 11, 2, 14593),
                                                (0, 11, 2, 19456), (0, 11, 2, 19457)])
def test_both_sides_of_the_one_thread_lines(ctx, model, box, camera, n):
    """32, 64 and 96 ROIs per SM, where one thread per ROI takes over, and 128, where
    its sCMOS blocks go from 128 ROIs to 96 (152 SMs): the bits of the shape set
    explicitly, and the oracle's results at the parity bar."""
    w = make_case(f"m{model}-{box}-{camera}", model, box, camera, n)
    got = run_gpu(ctx, w)
    line = 32 if box == 5 else 64 if box == 9 else 96
    shape = (4, 32) if n <= line * 152 else (1, 32 if not camera else 128 if n <= 128 * 152 else 96)
    ctx.check(ctx.lib.gmle_set_tuning(ctx.handle, model, box, camera, *shape))
    try:
        want = run_gpu(ctx, w)
    finally:
        ctx.check(ctx.lib.gmle_set_tuning(ctx.handle, model, box, camera, 0, 0))
    for a, b in zip(got, want):
        assert np.array_equal(a, b, equal_nan=True)
    if box > 5:
        check(w, got[0], got[1], got[3])


def test_table_launch_equals_plain(ctx):
    """A mixed submission below its line: the same warps, from a table."""
    torch = pytest.importorskip("torch")
    dev = torch.device("cuda", 0)
    ws = [make_case(f"m{m}-{b}", m, b, 0, n, seed=70 + b)
          for m, b, n in [(0, 4, 1), (0, 11, 200), (1, 16, 33), (2, 9, 301), (3, 15, 90)]]
    groups, outs = [], []
    for w in ws + ws:  # two groups of each kind
        data = torch.from_numpy(np.ascontiguousarray(w.data.transpose(2, 1, 0)).reshape(-1)).to(dev)
        P = w.psf.nparams
        o = [torch.empty((w.n, P), device=dev), torch.empty((w.n, P), device=dev),
             torch.empty(w.n, device=dev), torch.empty(w.n, dtype=torch.uint8, device=dev)]
        outs.append((w, data, o))
        groups.append(serve.make_group(w.psf, w.box, 0, w.constraints, data, None, None, *o))
    serve.fit_mixed_device(ctx, groups)
    torch.cuda.synchronize()
    for w, data, o in outs:
        p = [torch.empty_like(t) for t in o]
        G.fit_device(ctx, make_desc(w.psf, w.box, 20, w.constraints, 0), data, None, None, *p)
        torch.cuda.synchronize()
        for a, b in zip(o, p):
            assert torch.equal(a.nan_to_num(7.0), b.nan_to_num(7.0)), w.name


@pytest.mark.parametrize("model,camera,n", [(0, 2, 39_001), (3, 1, 39_137)])
def test_blocks_of_seven_warps(ctx, model, camera, n):
    """16x16 sCMOS batches from 256 ROIs per SM run in blocks of 224 ROIs, whose
    fifth to seventh warps keep their variances in a second set of tensor-memory
    columns: the same bits as in blocks of 128."""
    w = make_case(f"m{model}-16-{camera}", model, 16, camera, 500)
    rep = -(-n // w.n)
    w.data = np.asfortranarray(np.tile(w.data, (1, 1, rep))[:, :, :n])
    w.x_corners, w.y_corners = np.tile(w.x_corners, rep)[:n], np.tile(w.y_corners, rep)[:n]
    got = run_gpu(ctx, w)
    ctx.check(ctx.lib.gmle_set_tuning(ctx.handle, model, 16, camera, 1, 128))
    try:
        want = run_gpu(ctx, w)
    finally:
        ctx.check(ctx.lib.gmle_set_tuning(ctx.handle, model, 16, camera, 0, 0))
    for a, b in zip(got, want):
        assert np.array_equal(a, b, equal_nan=True)
