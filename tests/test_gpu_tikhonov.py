"""Tikhonov solves outside the right-hand-side kernel's tables (order 8, more
than 288 samples): by the operator product where H is well conditioned, by the
factor's substitutions elsewhere; and the L2 reference of the alpha path."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TIMES = dict(big_delta=0.043, small_delta=0.011)


def system(order, n_dirs, lam):
    """(bvals, bvecs, M, the regularization's diagonal, float32 signals)."""
    from cs_dmri_b200 import design_matrix
    from cs_dmri_b200.phantom import gradient_table, signals
    bvals, bvecs = gradient_table(1, n_dirs)
    M = design_matrix(bvals, bvecs, order, **TIMES)
    nl = [(n, l) for n in range(order + 1) for l in range(0, n + 1, 2) for _ in range(2 * l + 1)]
    reg = np.array([lam * (n * (n + 1)) ** 2 + lam * (l * (l + 1)) ** 2 for n, l in nl])
    return bvals, bvecs, M, reg, signals(5, np.arange(77), bvals, bvecs).astype(np.float32)


def gpu_fit(order, bvals, bvecs, s, lam):
    import torch
    from cs_dmri_b200.autograd import DifferentiableShore
    m = DifferentiableShore(bvals, bvecs, radial_order=order, regularization="l2", **TIMES)
    return m.fit(torch.from_numpy(s).cuda(), lambda_n=lam, lambda_l=lam).cpu().numpy()


@pytest.mark.parametrize("order,n_dirs,lam", [(8, 258, 0.0), (8, 514, 0.0), (8, 258, 1e-18), (8, 258, 1e-9),
                                              (8, 258, 1e-8), (6, 400, 0.0), (6, 400, 1e-8)])
def test_normal_equation_residual(order, n_dirs, lam):
    """Backward stable whatever the condition: rounding H and b costs N 2^-53
    |M|^T (|M| |c| + |s|) an entry, the solve K 2^-53 |H| |c|."""
    bvals, bvecs, M, reg, s = system(order, n_dirs, lam)
    c = gpu_fit(order, bvals, bvecs, s, lam)
    H, aM, ac = M.T @ M + np.diag(reg), np.abs(M), np.abs(c)
    N, K = M.shape
    bound = 2.0 ** -53 * (K * ac @ np.abs(H) + N * (ac @ aM.T @ aM + np.abs(s) @ aM))
    assert (np.abs(c @ H - s.astype(np.float64) @ M) <= bound).all()


def _substitutions(L, b):
    """L L^T x = b for the columns of b, in b's precision."""
    x = b.copy()
    for j in range(len(L)):
        x[j] /= L[j, j]
        x[j + 1:] -= np.outer(L[j + 1:, j], x[j])
    for j in range(len(L) - 1, -1, -1):
        x[j] /= L[j, j]
        x[:j] -= np.outer(L[j, :j], x[j])
    return x


@pytest.mark.parametrize("order,n_dirs", [(8, 258), (8, 150), (6, 400)])
@pytest.mark.parametrize("lam", [1e-8, 0.05])
def test_no_further_off_than_the_substitutions(order, n_dirs, lam):
    """Against the solution in extended precision, the median error is at most
    that of the factor's substitutions in float64 on b = M^T s summed as the
    kernels sum, one chain of fused multiply-adds in sample order."""
    bvals, bvecs, M, reg, s = system(order, n_dirs, lam)
    c = gpu_fit(order, bvals, bvecs, s, lam)
    ld = np.longdouble
    Ml, sl = M.astype(ld), s.astype(ld)
    A = Ml.T @ Ml + np.diag(reg.astype(ld))
    L = np.zeros_like(A)
    for j in range(len(A)):
        L[j:, j] = A[j:, j] / np.sqrt(A[j, j])
        A[j:, j:] -= np.outer(L[j:, j], L[j:, j])
    want = _substitutions(L, Ml.T @ sl.T).T
    L64 = np.linalg.cholesky(M.T @ M + np.diag(reg))
    b = np.zeros((len(s), M.shape[1]))
    for n in range(len(M)):  # a product and a sum of 64 bits, rounded to 53
        b = (b.astype(ld) + sl[:, n:n + 1] * Ml[n]).astype(np.float64)
    subst = _substitutions(L64, b.T).T

    def error(x):
        return float(np.median(np.linalg.norm((x - want).astype(float), axis=1) /
                               np.linalg.norm(want.astype(float), axis=1)))
    assert error(c) <= error(subst)


@pytest.mark.parametrize("order,lam", [(4, 1e-8), (6, 1e-8), (6, 0.0)])
@pytest.mark.parametrize("slack", [0.05, 0.0])
def test_host_and_device_paths_share_the_l2_reference(order, lam, slack):
    import torch
    from cs_dmri_b200 import shore_fit, shore_fit_device
    from test_gpu_sparse import tiled
    ph, data, mask = tiled(96)
    kw = dict(big_delta=ph.big_delta, small_delta=ph.small_delta, radial_order=order, alpha_mode="l2-anchored",
              lambda_n=lam, lambda_l=lam, slack=slack)
    host = shore_fit(data, ph.bvals, ph.bvecs, mask, **kw)["coefficients"]
    dev, _ = shore_fit_device(torch.from_numpy(np.ascontiguousarray(data)).cuda(), torch.from_numpy(mask).cuda(),
                              ph.bvals, ph.bvecs, **kw)
    np.testing.assert_array_equal(host, dev.cpu().numpy())


@pytest.mark.parametrize("lam", [1e-9, 0.05])  # by the substitutions, by the product
def test_a_refused_factor_leaves_no_trace(lam):
    """150 directions cannot determine 145 coefficients without a weight: the
    factor fails, and the fit with the earlier weight is what it was."""
    bvals, bvecs, _, _, s = system(8, 150, lam)
    want = gpu_fit(8, bvals, bvecs, s, lam)
    with pytest.raises(Exception, match="should be PD"):
        gpu_fit(8, bvals, bvecs, s, 0.0)
    np.testing.assert_array_equal(gpu_fit(8, bvals, bvecs, s, lam), want)
