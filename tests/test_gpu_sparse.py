"""The sparse FISTA kernel (one or two voxels per warp) against the DMMA
kernels and the oracle, at the sizes where its dispatch and its slots change.

Every FP64 FISTA kernel adds the same products in the same order and shares
the update, so coefficients, iteration counts and flags are compared bit for
bit; the oracle comparison uses the parity bounds (coefficients 1e-5 per
voxel, iterations within 1: a stopping decision within rounding of tol).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("coef64", "coefficients", "iterations", "converged")


def tiled(v, seed=41):
    """A (v, 1, 1) volume that repeats 96 phantom voxels (the last one zero)."""
    from cs_dmri_b200.phantom import make_phantom
    ph = make_phantom((12, 8, 1), seed=seed)
    rows = ph.data.reshape(96, -1).copy()
    rows[95] = 0.0
    data = rows[np.arange(v) % 96].reshape(v, 1, 1, -1)
    return ph, data, np.ones((v, 1, 1), bool)


def fit(ph, data, mask, **kw):
    from cs_dmri_b200 import shore_fit
    return shore_fit(data, ph.bvals, ph.bvecs, mask, big_delta=ph.big_delta, small_delta=ph.small_delta,
                     return_coef64=True, diagnostics=True, **kw)


@pytest.mark.parametrize("order", [4, 6])
@pytest.mark.parametrize("v", [1, 33, 601, 16577, 18943, 18944, 19001])
@pytest.mark.parametrize("kw", [dict(alpha_mode="fixed", alpha=0.01),
                                dict(alpha_mode="fixed", alpha=0.02, non_negative=True, max_iter=37),
                                dict(alpha_mode="alpha-ratio", alpha_ratio=0.01)])
def test_matches_the_dmma_kernel_bit_for_bit(order, v, kw):
    """Order 6: two voxels per warp from 16,577; from 18,944 (one wave of DMMA
    slots) the first 80 iterations run on those and the rest on sparse warps.
    """
    from cs_dmri_b200 import _abi
    ph, data, mask = tiled(v)
    sparse = fit(ph, data, mask, radial_order=order, **kw)
    _abi.set_option(_abi.OPT_FISTA_SHAPE, 16)
    try:
        dmma = fit(ph, data, mask, radial_order=order, **kw)
    finally:
        _abi.set_option(_abi.OPT_FISTA_SHAPE, 0)
    for k in KEYS:
        np.testing.assert_array_equal(sparse[k], dmma[k])


@pytest.mark.parametrize("v", [14209, 14304])  # two voxels per warp from 14,209
def test_order_8_two_voxels_per_warp_equal_one(v, oracle):
    ph, data, mask = tiled(v)
    two = fit(ph, data, mask, radial_order=8, alpha_mode="fixed", alpha=0.01)
    one = fit(ph, data[:96], mask[:96], radial_order=8, alpha_mode="fixed", alpha=0.01)
    at = np.arange(v) % 96
    np.testing.assert_array_equal(two["coef64"], one["coef64"][at])
    np.testing.assert_array_equal(two["converged"], one["converged"][at])
    np.testing.assert_array_equal(two["iterations"].ravel(), one["iterations"].ravel()[at])
    ref = oracle.shore_fit(data[:96], ph.bvals, ph.bvecs, mask[:96], big_delta=ph.big_delta,
                           small_delta=ph.small_delta, radial_order=8, alpha_mode="fixed", alpha=0.01,
                           diagnostics=True)
    num = np.linalg.norm(one["coef64"] - ref["coef64"], axis=1)
    assert (num <= 1e-5 * np.linalg.norm(ref["coef64"], axis=1)).all()
    assert np.abs(one["iterations"].astype(int) - ref["iterations"].astype(int)).max() <= 1


@pytest.mark.parametrize("order,v", [(6, 5), (6, 2400), (6, 9475), (4, 9475), (8, 40)])
@pytest.mark.parametrize("mode", ["l2-anchored", "path-bic"])
def test_fused_path_equals_the_path_point_by_point(order, v, mode):
    """Sizes of the fused path's three forms at order 6 (one and two voxels
    per warp; from 9,472 the DMMA slots, which hand their last voxels over).
    The residuals behind the selection are summed in another order (relative
    1e-15), so a selection within that of a tie could differ; none does here.
    """
    from cs_dmri_b200 import _abi
    ph, data, mask = tiled(v)
    kw = dict(radial_order=order, alpha_mode=mode, path_n_alphas=9)
    fused = fit(ph, data, mask, **kw)
    _abi.set_option(_abi.OPT_FISTA_SHAPE, 16)  # a forced shape walks the path point by point
    try:
        walk = fit(ph, data, mask, **kw)
    finally:
        _abi.set_option(_abi.OPT_FISTA_SHAPE, 0)
    for k in KEYS + ("alpha",):
        np.testing.assert_array_equal(fused[k], walk[k])
    for k in ("bic", "r2", "residual_l2"):
        np.testing.assert_allclose(fused[k], walk[k], rtol=1e-6, atol=1e-6)
    assert fused["total_iterations"] == walk["total_iterations"]
