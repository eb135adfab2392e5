"""One warp per ROI (boxes 17..64): the edges of its lane grid.

A lane owns every 8th column and every 4th row, in register slots up to box 32
and from shared memory beyond, and a block takes up to four ROIs: boxes at and
next to the multiples of 4 and 8 and the borders of the compiled ranges (17,
20/21, 24/25, 28/29, 32/33, 48/49, 64), with batches that leave warps empty.
Compared with the oracle at the parity bar (test_boxes_gpu.check)."""
import numpy as np
import pytest

from gaussmle_gb300.fitter import make_desc
from oracle import oracle as O
from parity_cases import make_case, oracle_desc
from test_boxes_gpu import check
from test_edge_gpu import host_fit, set_maps
from test_parity_gpu import run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,camera", [(0, 0), (1, 2), (2, 1), (2, 0)])
@pytest.mark.parametrize("box,n", [(17, 1), (20, 3), (25, 6), (28, 4), (29, 9), (31, 2), (32, 5),
                                   (33, 3), (48, 7), (49, 2), (63, 5), (64, 3)])
def test_lane_grid_edges(ctx, model, camera, box, n):
    w = make_case(f"m{model}-{box}-{camera}", model, box, camera, n)
    params, crlb, llr, flags = run_gpu(ctx, w)
    check(w, params, crlb, flags)
    ref = O.fit(oracle_desc(O, w), w.data, w.x_corners, w.y_corners, w.maps, "f64")
    # the LLR's FP32 sums: box^2 terms of size |LLR| / box^2 and, for Poisson
    # data, differences of logarithm terms of size d ln d (to 3e-7 absolute each)
    scale = np.abs(ref["llr"]) + (0 if camera else w.data.reshape(box * box, n).sum(0) * 0.5)
    assert np.all(np.abs(llr - ref["llr"]) <= 1e-4 * scale)


@pytest.mark.parametrize("model,box,camera", [(0, 17, 0), (1, 32, 2), (3, 33, 0), (3, 21, 2)])
def test_start_point(ctx, model, box, camera):
    """No iterations: the start point, whose sums run over the lanes.  A lane
    adds at most 128 pixels, 5 more additions join the lanes, and x, y and z
    are quotients of two such sums: 2 * 133 * 2^-24 relative."""
    w = make_case(f"m{model}-{box}-{camera}", model, box, camera, 11)
    if w.camera:
        set_maps(ctx, w.maps)
    desc = make_desc(w.psf, box, 0, w.constraints, camera)
    st, (prm, *_) = host_fit(ctx, desc, w.data, w.x_corners, w.y_corners)
    ctx.check(st)
    ref = O.fit(oracle_desc(O, w, iterations=0), w.data, w.x_corners, w.y_corners, w.maps, "f64")
    keep = [k for k in range(prm.shape[1]) if not (model == 3 and k == 2)]
    np.testing.assert_allclose(prm[:, keep], ref["params"][:, keep], rtol=1.6e-5)
    if model == 3:  # z: a difference of two squared width ratios, times d^2 / (4 gamma) = 50
        np.testing.assert_allclose(prm[:, 2], ref["params"][:, 2], rtol=0,
                                   atol=50 * 4 * 1.6e-5 * box)
