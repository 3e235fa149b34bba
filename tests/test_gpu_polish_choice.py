"""The first polish of the converged-optimum modes above 384 voxels per SM:
two voxels per warp where few starting supports hold more than sixteen
coefficients, one elsewhere, against the form that serves smaller fits (one).

Tolerances as in the polish's own test: both forms factorise the same support
with the same operations in the same order and stop at the certified minimiser,
so coefficients agree to 1e-12.  The starting iterate in FP64 shares its memory
with the result, so voxels left to the second launch must be untouched.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [4, 6])
@pytest.mark.parametrize("precision", ["mixed-kkt", "fp64-kkt"])
@pytest.mark.parametrize("kw", [dict(alpha_mode="fixed", alpha=0.01), dict(alpha_mode="fixed", alpha=0.008),
                                dict(alpha_mode="fixed", alpha=0.002), dict(alpha_mode="alpha-ratio", alpha_ratio=0.03),
                                dict(alpha_mode="fixed", alpha=0.01, non_negative=True)])
def test_large_fits_equal_small_ones(order, precision, kw):
    from cs_dmri_b200 import shore_fit
    from cs_dmri_b200.phantom import make_phantom
    v = 56849
    ph = make_phantom((12, 8, 1), seed=29)
    rows = ph.data.reshape(96, -1).copy()
    rows[95, 7] = np.nan  # zero coefficients, not certified
    at = np.arange(v) % 96

    def fit(which):
        data = np.ascontiguousarray(rows[which].reshape(len(which), 1, 1, -1))
        return shore_fit(data, ph.bvals, ph.bvecs, np.ones((len(which), 1, 1), bool), big_delta=ph.big_delta,
                         small_delta=ph.small_delta, radial_order=order, precision=precision, return_coef64=True,
                         diagnostics=True, **kw)

    small, large = fit(np.arange(96)), fit(at)
    np.testing.assert_array_equal(large["converged"].ravel(), small["converged"].ravel()[at])
    # alpha_max of the NaN voxel is 0, so under alpha-ratio it has the zero result, converged
    assert small["converged"].sum() == (95 if kw["alpha_mode"] == "fixed" else 96)
    err = np.linalg.norm(large["coef64"] - small["coef64"][at], axis=1)
    assert (err <= 1e-12 * np.linalg.norm(small["coef64"][at], axis=1)).all()
    assert (large["iterations"].ravel() == small["iterations"].ravel()[at]).mean() >= 0.99
