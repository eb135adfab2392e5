"""The p-values' table (gmle_pvalue.cu): degrees of freedom on both sides of the
lines where it is used (16) and where its spacing changes (32), the largest
boxes' and beyond, and the ends of its node range, against the reference's
formula.  A Float32 cdf rounded from a value within 1e-9 of the exact one is
within one ulp of 1 of the formula's."""
import numpy as np
import pytest

from oracle import oracle as O
from test_pvalues_gpu import TOL, _gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("df", [15, 16, 17, 31, 32, 33, 63, 64, 65, 1020, 4092, 100_000])
@pytest.mark.parametrize("n", [1, 511, 513, 30_000])
def test_table_matches_the_reference_formula(ctx, df, n):
    rng = np.random.default_rng(df + n)
    chi2 = np.concatenate([rng.chisquare(df, n),
                           df + np.sqrt(2.0 * df) * np.linspace(-12, 16, n)]).astype(np.float32)
    llr = (-0.5 * chi2).astype(np.float32)
    np.testing.assert_allclose(_gpu(ctx, llr, df), O.pvalues(llr, df), rtol=0, atol=TOL)


@pytest.mark.parametrize("df", [16, 117])
def test_special_values(ctx, df):
    llr = np.array([np.nan, np.inf, -np.inf, 0.0, -0.0, 1e30, -1e30, -3e9, -1e-38], np.float32)
    want = np.array([np.nan, 1, 0, 1, 1, 1, 0, 0, 1], np.float32)
    np.testing.assert_array_equal(_gpu(ctx, llr, df), want)
