"""Per-voxel designs at the ends of their ranges: no and few iterations, and
voxels without samples between full ones."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def inputs():
    from cs_dmri_b200.graddev import graddev_phantom
    return graddev_phantom(24, seed=11)


@pytest.mark.parametrize("order", [6, 8])
@pytest.mark.parametrize("max_iter", [0, 1, 2])
@pytest.mark.parametrize("non_negative", [False, True])
def test_few_iterations_match_the_oracle(oracle, inputs, order, max_iter, non_negative):
    """Coefficients within 1e-10 of the largest: a few steps of the same update,
    whose step size agrees to 1e-12."""
    from cs_dmri_b200.graddev import shore_fit_graddev
    S, bvals, bvecs, T, keep, big, small = inputs
    kw = dict(radial_order=order, big_delta=big, small_delta=small, max_iter=max_iter, non_negative=non_negative)
    out = shore_fit_graddev(S, bvals, bvecs, T, keep, alpha=0.01, **kw)
    c, it = out["coefficients"].cpu().numpy(), out["iterations"].cpu().numpy()
    for v in range(0, len(S), 5):
        want, wit, wconv, _ = oracle.graddev_fit(S[v], bvals, bvecs, T[v], keep[v], 0.01, **kw)
        np.testing.assert_allclose(c[v], want, rtol=0, atol=1e-10 * max(np.abs(want).max(), 1e-300))
        assert it[v] == wit == max_iter and bool(out["converged"][v]) == wconv


@pytest.mark.parametrize("order", [6, 8])
@pytest.mark.parametrize("precision", ["fp64", "fp64-kkt", "mixed-kkt"])
def test_a_voxel_without_samples_stays_alone(inputs, order, precision):
    from cs_dmri_b200.graddev import shore_fit_graddev
    S, bvals, bvecs, T, keep, big, small = inputs
    kw = dict(alpha=0.01, radial_order=order, big_delta=big, small_delta=small, precision=precision)
    want = shore_fit_graddev(S, bvals, bvecs, T, keep, **kw)
    none = keep.copy()
    none[[0, 7, 23]] = False
    got = shore_fit_graddev(S, bvals, bvecs, T, none, **kw)
    full = np.ones(24, bool)
    full[[0, 7, 23]] = False
    for k in ("coefficients", "iterations", "converged", "lipschitz"):
        np.testing.assert_array_equal(got[k].cpu().numpy()[full], want[k].cpu().numpy()[full])
    assert not bool(got["coefficients"][~full].any()) and int(got["n_samples"][~full].sum()) == 0
