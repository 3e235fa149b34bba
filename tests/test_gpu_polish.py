"""The converged-optimum polish with two voxels per warp (above 384 voxels
per SM) against the form with one, which serves smaller fits.

Both factorise the same support with the same operations in the same order,
and both stop at the certified minimiser; coefficients are compared at 1e-12
relative (the gradient's last bits could take another coordinate first), round
counts exactly up to 1 % of the voxels.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("v", [56833, 56849])
@pytest.mark.parametrize("kw", [dict(alpha=0.01), dict(alpha=0.0005), dict(alpha=0.01, non_negative=True)])
def test_two_voxels_per_warp_equal_one(order, v, kw):
    from cs_dmri_b200 import shore_fit
    from cs_dmri_b200.phantom import make_phantom
    ph = make_phantom((12, 8, 1), seed=23)
    rows = ph.data.reshape(96, -1).copy()
    rows[94] = 0.0             # an empty support
    rows[95, 7] = np.nan       # zero coefficients, not certified
    at = np.arange(v) % 96

    def fit(which):
        data = np.ascontiguousarray(rows[which].reshape(len(which), 1, 1, -1))
        return shore_fit(data, ph.bvals, ph.bvecs, np.ones((len(which), 1, 1), bool), big_delta=ph.big_delta,
                         small_delta=ph.small_delta, radial_order=order, alpha_mode="fixed", precision="mixed-kkt",
                         return_coef64=True, diagnostics=True, **kw)

    one, two = fit(np.arange(96)), fit(at)
    np.testing.assert_array_equal(two["converged"].ravel(), one["converged"].ravel()[at])
    assert one["converged"].sum() == 95
    err = np.linalg.norm(two["coef64"] - one["coef64"][at], axis=1)
    assert (err <= 1e-12 * np.linalg.norm(one["coef64"][at], axis=1)).all()
    assert (two["iterations"].ravel() == one["iterations"].ravel()[at]).mean() >= 0.99
