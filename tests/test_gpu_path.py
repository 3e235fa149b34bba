"""The fused alpha path beyond its defaults: non-negative fits, few iterations,
voxels that are not finite, and its counters.

As in the fused path's own test, every kernel shares the update and the order
of its sums, so coefficients, iteration counts, flags and alphas equal those of
the path walked point by point bit for bit; only the residuals behind the
selection are summed in another order (1e-15 relative).
"""

import numpy as np
import pytest

from test_gpu_sparse import KEYS, fit, tiled

pytestmark = pytest.mark.gpu


def walked(ph, data, mask, **kw):
    from cs_dmri_b200 import _abi
    _abi.set_option(_abi.OPT_FISTA_SHAPE, 16)  # a forced shape walks the path point by point
    try:
        return fit(ph, data, mask, **kw)
    finally:
        _abi.set_option(_abi.OPT_FISTA_SHAPE, 0)


@pytest.mark.parametrize("order,v", [(6, 5), (6, 2400), (6, 9475), (4, 2400), (4, 9475), (8, 40)])
@pytest.mark.parametrize("mode", ["l2-anchored", "path-bic"])
@pytest.mark.parametrize("kw", [dict(non_negative=True), dict(max_iter=1), dict(max_iter=60, non_negative=True)])
def test_fused_path_equals_the_walk(order, v, mode, kw):
    ph, data, mask = tiled(v)
    kw = dict(radial_order=order, alpha_mode=mode, path_n_alphas=7, **kw)
    fused, walk = fit(ph, data, mask, **kw), walked(ph, data, mask, **kw)
    for k in KEYS + ("alpha",):
        np.testing.assert_array_equal(fused[k], walk[k])
    assert fused["total_iterations"] == walk["total_iterations"]


@pytest.mark.parametrize("v", [300, 2400, 9475])
@pytest.mark.parametrize("mode", ["l2-anchored", "path-bic"])
def test_voxels_that_are_not_finite_stay_alone(v, mode):
    ph, data, mask = tiled(v)
    kw = dict(radial_order=6, alpha_mode=mode, path_n_alphas=7)
    want = fit(ph, data, mask, **kw)
    bad = data.copy()
    at = [1, v // 2, v - 2]
    for i, value in zip(at, (np.nan, np.inf, -np.inf)):
        bad[i, 0, 0, 9] = value
    got = fit(ph, bad, mask, **kw)
    keep = np.ones(v, bool)
    keep[at] = False
    for k in KEYS + ("alpha",):
        np.testing.assert_array_equal(got[k].reshape(v, -1)[keep], want[k].reshape(v, -1)[keep])
    assert not got["coef64"][1].any()  # alpha_max of a NaN right-hand side is 0


@pytest.mark.parametrize("order,v", [(6, 11000), (6, 19001), (4, 12000)])
def test_two_passes_leave_finite_voxels_alone(order, v):
    ph, data, mask = tiled(v)
    kw = dict(radial_order=order, alpha_mode="fixed", alpha=0.005)
    want = fit(ph, data, mask, **kw)
    bad = data.copy()
    bad[3, 0, 0, 9], bad[v - 3, 0, 0, 0] = np.nan, np.inf
    got = fit(ph, bad, mask, **kw)
    keep = np.ones(v, bool)
    keep[[3, v - 3]] = False
    for k in KEYS:
        np.testing.assert_array_equal(got[k].reshape(v, -1)[keep], want[k].reshape(v, -1)[keep])


def test_the_path_on_dmma_slots_counts_its_tensor_operations():
    from cs_dmri_b200 import _abi
    ph, data, mask = tiled(9475)
    out = fit(ph, data, mask, radial_order=6, alpha_mode="l2-anchored", path_n_alphas=7)
    dense = 2.0 * 72 * 72 * out["total_iterations"]  # live k-steps only, and slots left empty
    assert 0.1 * dense < _abi.last_timing(0).tensor_flops < 1.5 * dense


@pytest.mark.parametrize("order", [2, 6])
def test_a_path_without_a_finite_residual_gives_zero(order):
    """The walk and the fused path alike; the walk's scratch holds another fit's
    fallback points from the call before."""
    ph, data, mask = tiled(96)
    kw = dict(radial_order=order, alpha_mode="l2-anchored", path_n_alphas=5, slack=0.0)
    run = walked if order == 6 else fit
    run(ph, data, mask, **kw)
    bad = data.copy()
    bad[40, 0, 0, 9] = np.inf
    for out in (run(ph, bad, mask, **kw), fit(ph, bad, mask, **kw)):
        assert not out["coef64"][40].any() and out["alpha"].ravel()[40] == 0.0
        assert out["iterations"].ravel()[40] == 0 and out["converged"].ravel()[40]
