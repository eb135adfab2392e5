"""The rounding of Poisson fits.  Their log-likelihood ratio sums d ln mu - mu -
(d ln d - d), thousands in a bright pixel and rounded to some 1e-4 before they
cancel, so that its error, and 2e-5 of a small box's p-values, hangs on the last bits
of mu and of the fitted parameters.  poisson_rounding.npz holds the fits (one thread
per ROI and four lanes) of the kernels that evaluate each pixel edge's erf at
(t + 1/2 - c) * sqrt(1/2 / sigma^2) and d / mu rounded before 1 is subtracted.

Bounds: parameters that carry the same rounding differ only where the Hessian's last
bits or an FMA of a width's derivative change a step, in at most a tenth of the XYNB
fits, a third of the XYNBS ones and half of the ill-conditioned astigmatic ones (with
another rounding of the edges, or of d / mu, nine and four tenths of the XYNB fits
do); from the same parameters comes the same ratio, but for a sum's last bits (and
the few pixels where t - c itself rounds); and the p-values are within 32-bit
rounding of the bright pixels, 2e-5 of their norm."""
from pathlib import Path

import numpy as np
import pytest

from oracle import oracle as O
from parity_cases import make_case
from test_parity_gpu import run_gpu

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden" / "poisson_rounding.npz"


@pytest.mark.parametrize("tpr", [1, 4])
@pytest.mark.parametrize("model,box,same", [(0, 7, 0.9), (1, 7, 0.66), (3, 13, 0.5)])
def test_parameters_and_ratio_keep_their_rounding(ctx, model, box, same, tpr):
    g = np.load(GOLDEN)
    key = f"m{model}_{box}_"
    data = g[key + "data"].astype(np.float32)
    w = make_case(f"m{model}-{box}", model, box, 0, data.shape[2])
    w.data = np.asfortranarray(data)
    ctx.check(ctx.lib.gmle_set_tuning(ctx.handle, model, box, 0, tpr, 32))
    try:
        params, _, llr, _ = run_gpu(ctx, w)
    finally:
        ctx.check(ctx.lib.gmle_set_tuning(ctx.handle, model, box, 0, 0, 0))
    want, want_llr = g[key + f"params{tpr}"], g[key + f"llr{tpr}"]
    equal = (params == want).all(1)
    assert equal.mean() >= same
    near = np.abs(llr - want_llr)[equal] <= 1e-6 * np.abs(want_llr[equal])
    assert near.mean() >= 0.98
    df = box * box - params.shape[1]
    p, q = O.pvalues(llr, df).astype(float), O.pvalues(want_llr, df).astype(float)
    assert np.linalg.norm(p - q) <= 2e-5 * np.linalg.norm(q)
