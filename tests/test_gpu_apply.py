"""The fixed-matrix product on the tensor cores at the edges of its tiles and
row chunks, and the Tikhonov solves built on it."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 1), (8, 4), (9, 5), (97, 96), (72, 362), (362, 145), (145, 362), (515, 72),
                                       (104, 3632)])  # the widest matrix admitted
@pytest.mark.parametrize("v", [1, 9, 300, 2500])
def test_apply_matches_the_product(rows, cols, v):
    """Each output is one FMA chain over cols terms: its error is at most
    cols 2^-53 sum |a| |x|, and the float64 matmul's the same again."""
    import torch
    from cs_dmri_b200.autograd import DifferentiableShore
    from cs_dmri_b200.phantom import gradient_table
    m = DifferentiableShore(*gradient_table(1), big_delta=0.043, small_delta=0.011)
    gen = torch.Generator(device="cuda").manual_seed(rows * 7919 + cols + v)
    f64 = dict(dtype=torch.float64, device="cuda", generator=gen)
    A, x = torch.randn((rows, cols), **f64), torch.randn((v, cols), **f64)
    x[v // 2] = float("nan")  # one voxel's NaN stays its own
    got = m._apply_raw(A.T.contiguous(), rows, cols, x)
    keep = torch.arange(v, device="cuda") != v // 2
    assert bool(got[v // 2].isnan().all())
    want, bound = x[keep] @ A.T, x[keep].abs() @ A.abs().T
    assert bool(((got[keep] - want).abs() <= 2 * cols * 2.0 ** -53 * bound).all())
    if cols == 3632:
        with pytest.raises(ValueError, match="too wide"):
            m._apply_raw(torch.zeros((3633, 2), dtype=torch.float64, device="cuda"), 2, 3633, x)


@pytest.mark.parametrize("order,n_dirs,lam", [(8, 258, 0.05), (8, 150, 1e-8), (8, 514, 0.01), (6, 400, 0.05)])
def test_tikhonov_by_the_refined_inverse(order, n_dirs, lam):
    """Order 8 and tables past 288 samples: normal-equation residual of a
    backward stable solve, K 2^-53 (|H| |c| + |b|) per entry."""
    import torch
    from cs_dmri_b200 import design_matrix
    from cs_dmri_b200.autograd import DifferentiableShore
    from cs_dmri_b200.phantom import gradient_table, signals
    bvals, bvecs = gradient_table(1, n_dirs)
    kw = dict(big_delta=0.043, small_delta=0.011)
    m = DifferentiableShore(bvals, bvecs, radial_order=order, regularization="l2", **kw)
    s = torch.from_numpy(signals(5, np.arange(77), bvals, bvecs)).cuda()
    c = m.fit(s, lambda_n=lam, lambda_l=lam).cpu().numpy()
    M = design_matrix(bvals, bvecs, order, **kw)
    nl = [(n, l) for n in range(order + 1) for l in range(0, n + 1, 2) for _ in range(2 * l + 1)]
    H = M.T @ M + np.diag([lam * (n * (n + 1)) ** 2 + lam * (l * (l + 1)) ** 2 for n, l in nl])
    b = s.cpu().numpy().astype(np.float64) @ M
    bound = np.abs(c) @ np.abs(H) + np.abs(b) + np.abs(s.cpu().numpy()) @ np.abs(M)
    assert (np.abs(c @ H - b) <= len(nl) * 2.0 ** -53 * bound).all()


@pytest.mark.parametrize("order", [2, 6, 8])
@pytest.mark.parametrize("v", [1, 7, 8, 9, 16, 17, 2385])
def test_predicted_signal_at_ragged_volumes(order, v, oracle):
    """Eight voxels a thread, sixteen a tile: every sum is in coefficient
    order without fused operations, so the signals equal the oracle's to one
    rounding of a design entry per term; zero voxels stay zero."""
    from cs_dmri_b200 import shore_predict
    from cs_dmri_b200.phantom import make_phantom
    ph = make_phantom((2, 2, 2), seed=5)
    K = sum(2 * l + 1 for n in range(order + 1) for l in range(0, n + 1, 2))
    rng = np.random.default_rng(v)
    c = rng.normal(size=(v, 1, 1, K)).astype(np.float32)
    c[v // 2] = 0.0
    kw = dict(big_delta=ph.big_delta, small_delta=ph.small_delta)
    got = shore_predict(c, order, 700.0, ph.bvals, ph.bvecs, **kw)
    want = oracle.shore_predict(c, order, 700.0, ph.bvals, ph.bvecs, **kw)
    assert not got[v // 2].any()
    scale = np.abs(want).max()
    np.testing.assert_allclose(got, want, rtol=2.4e-7, atol=1e-9 * max(scale, 1e-30))
