"""The rounding of an sCMOS fit's log-likelihood ratio, a sum over all pixels: with one
thread per ROI its error is no larger than with four lanes, whose sums are a quarter
as long.  Reference: the same ratio in 64 bits at the parameters that the fit returned.

Bound: each rounding of a running sum adds a term of 2^-24 of it, so that the sums' error
grows with the root of the longest sum's length: 169 pixels in one sum is twice
sqrt(43), 13 sums of 13 pixels added up about half of it.  5 % for the sample (2 000
ROIs)."""
import numpy as np
import pytest
from scipy.special import erf

from parity_cases import make_case
from test_edge_gpu import set_maps
from test_parity_gpu import run_gpu

pytestmark = pytest.mark.gpu


def ratio64(w, params):
    p = params.astype(np.float64)
    t = np.arange(1, w.box + 1)

    def psf(c, s):
        u = lambda e: (e[None, :] - c[:, None]) / (np.sqrt(2) * s[:, None])
        return 0.5 * (erf(u(t + 0.5)) - erf(u(t - 0.5)))

    mu = p[:, 3, None, None] + p[:, 2, None, None] * (psf(p[:, 0], p[:, 4])[:, :, None] *
                                                      psf(p[:, 1], p[:, 4])[:, None, :])
    rows = w.y_corners[:, None, None] - 1 + np.arange(w.box)[None, None, :]
    cols = w.x_corners[:, None, None] - 1 + np.arange(w.box)[None, :, None]
    v = w.maps[0][rows, cols].astype(np.float64)
    d = w.data.transpose(2, 1, 0).astype(np.float64)
    return (-0.5 * (d - mu) ** 2 / (mu + v)).sum((1, 2))


@pytest.mark.parametrize("box", [13, 15])
def test_one_thread_sums_as_exactly_as_four_lanes(ctx, box):
    w = make_case(f"m1-{box}-1", 1, box, 1, 2000)
    set_maps(ctx, w.maps)
    error = {}
    for shape in ((1, 128), (4, 32)):
        ctx.check(ctx.lib.gmle_set_tuning(ctx.handle, 1, box, 1, *shape))
        try:
            params, _, llr, _ = run_gpu(ctx, w)
        finally:
            ctx.check(ctx.lib.gmle_set_tuning(ctx.handle, 1, box, 1, 0, 0))
        want = ratio64(w, params)
        error[shape[0]] = np.linalg.norm(llr - want) / np.linalg.norm(want)
    assert error[4] < 1e-6
    assert error[1] <= 1.05 * error[4], error
