"""A refused amplitude-positivity setup leaves no trace in later fits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1])  # Gram form, basis form (which keeps the factor)
def test_a_refused_setup_leaves_no_trace(form):
    """51 samples cannot determine 72 coefficients without epsilon: the factor
    fails, and the fit with the earlier epsilon is what it was."""
    from cs_dmri_b200 import _abi, shore_fit
    from cs_dmri_b200.phantom import gradient_table, signals
    bvals, bvecs = gradient_table(1, 50)
    data = signals(5, np.arange(20), bvals, bvecs).astype(np.float32).reshape(20, 1, 1, -1)
    kw = dict(big_delta=0.043, small_delta=0.011, radial_order=6, regularization="nonneg", return_coef64=True)
    mask = np.ones((20, 1, 1), bool)
    _abi.set_option(_abi.OPT_ICLS, form)
    try:
        want = shore_fit(data, bvals, bvecs, mask, nonneg_epsilon=1e-6, **kw)["coef64"]
        with pytest.raises(Exception, match="positive definite"):
            shore_fit(data, bvals, bvecs, mask, nonneg_epsilon=-1e-3, **kw)
        np.testing.assert_array_equal(shore_fit(data, bvals, bvecs, mask, nonneg_epsilon=1e-6, **kw)["coef64"], want)
    finally:
        _abi.set_option(_abi.OPT_ICLS, 0)
