"""The Gram form of the amplitude-positivity fit at the edges of its grid (20
warps a CTA, one CTA an SM) and of its active sets, against the
orthogonal-basis form.

The two forms walk the same iteration path and differ by rounding, so the
bounds are those of the parity tests: coefficients 1e-8 (median) and 1e-5 per
voxel; iteration counts equal except where a rounding decides (1 % of voxels).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("v", [1, 20, 21, 2961])
@pytest.mark.parametrize("kw", [{}, dict(nonneg_max_iter=0), dict(nonneg_max_iter=3)])
def test_gram_form_equals_the_basis_form(order, v, kw):
    from cs_dmri_b200 import _abi, shore_fit
    from cs_dmri_b200.phantom import make_phantom
    ph = make_phantom((8, 6, 1), seed=17)
    rows = ph.data.reshape(48, -1).copy()
    rng = np.random.default_rng(3)
    rows[24:] = np.abs(rows[24:] + rng.normal(0.0, 0.3 * rows[24:].mean(), rows[24:].shape))  # many active constraints
    rows[47] = 0.0
    data = np.ascontiguousarray(rows[(np.arange(v) + 20) % 48].reshape(v, 1, 1, -1).astype(np.float32))
    mask = np.ones((v, 1, 1), bool)
    out = []
    for form in (0, 1):
        _abi.set_option(_abi.OPT_ICLS, form)
        try:
            out.append(shore_fit(data, ph.bvals, ph.bvecs, mask, big_delta=ph.big_delta, small_delta=ph.small_delta,
                                 regularization="nonneg", radial_order=order, return_coef64=True, diagnostics=True,
                                 **kw))
        finally:
            _abi.set_option(_abi.OPT_ICLS, 0)
    gram, basis = out
    same = gram["iterations"].ravel() == basis["iterations"].ravel()
    assert same.mean() >= 0.99
    np.testing.assert_array_equal(gram["converged"].ravel()[same], basis["converged"].ravel()[same])
    err = np.linalg.norm(gram["coef64"] - basis["coef64"], axis=1)
    err = err[same] / np.maximum(np.linalg.norm(basis["coef64"], axis=1)[same], 1e-12)
    assert np.median(err) <= 1e-8 and err.max() <= 1e-5
