"""Fits whose iterates are dense (small alpha): the second pass of a fit goes
to the DMMA slots where the parked voxels' momentum points have many non-zero
entries, to sparse warps elsewhere.

Every FP64 FISTA kernel computes the same iterates, so results are compared
bit for bit with the DMMA kernel's.  The route shows in the executed FP64
tensor operations of two fits that differ in their last iterations only: a
second pass on DMMA slots executes more of them when max_iter grows from 161 to
1,000, one on sparse warps none beyond the first 80 iterations (up to the
products of partly filled slots, which depend on timing).
"""

import numpy as np
import pytest

from test_gpu_sparse import KEYS, fit, tiled

pytestmark = pytest.mark.gpu


def tensor_growth(ph, data, mask, **kw):
    """Executed tensor operations with max_iter 1,000 over those with 161."""
    from cs_dmri_b200 import _abi
    flops = []
    for max_iter in (161, 1000):
        fit(ph, data, mask, max_iter=max_iter, **kw)
        flops.append(_abi.last_timing(0).tensor_flops)
    assert flops[0] > 0.0
    return flops[1] / flops[0]


@pytest.mark.parametrize("order,v", [(4, 11839), (4, 11840), (4, 25001), (6, 8287), (6, 8288), (6, 10655),
                                     (6, 10656), (6, 19001)])
@pytest.mark.parametrize("kw", [dict(alpha_mode="fixed", alpha=0.001), dict(alpha_mode="alpha-ratio"),
                                dict(alpha_mode="fixed", alpha=0.0005, non_negative=True, max_iter=200)])
def test_dense_fits_match_the_dmma_kernel_bit_for_bit(order, v, kw):
    from cs_dmri_b200 import _abi
    ph, data, mask = tiled(v)
    chosen = fit(ph, data, mask, radial_order=order, **kw)
    _abi.set_option(_abi.OPT_FISTA_SHAPE, 16)
    try:
        dmma = fit(ph, data, mask, radial_order=order, **kw)
    finally:
        _abi.set_option(_abi.OPT_FISTA_SHAPE, 0)
    for k in KEYS:
        np.testing.assert_array_equal(chosen[k], dmma[k])


@pytest.mark.parametrize("order,v", [(4, 7103), (4, 7104), (4, 11839), (4, 11840), (6, 5327), (6, 5328), (6, 8287),
                                     (6, 8288)])
@pytest.mark.parametrize("max_iter", [20, 160, 161])
@pytest.mark.parametrize("alpha", [0.0005, 0.02])
def test_short_fits_match_the_dmma_kernel_bit_for_bit(order, v, max_iter, alpha):
    from cs_dmri_b200 import _abi
    ph, data, mask = tiled(v)
    kw = dict(radial_order=order, alpha_mode="fixed", alpha=alpha, max_iter=max_iter)
    chosen = fit(ph, data, mask, **kw)
    _abi.set_option(_abi.OPT_FISTA_SHAPE, 12)
    try:
        dmma = fit(ph, data, mask, **kw)
    finally:
        _abi.set_option(_abi.OPT_FISTA_SHAPE, 0)
    for k in KEYS:
        np.testing.assert_array_equal(chosen[k], dmma[k])


@pytest.mark.parametrize("order,v", [(4, 20000), (4, 25001), (4, 25056), (6, 15000), (6, 20000), (6, 76000)])
def test_the_second_pass_follows_the_density(order, v):
    ph, data, mask = tiled(v)
    assert tensor_growth(ph, data, mask, radial_order=order, alpha_mode="alpha-ratio") > 1.5
    assert tensor_growth(ph, data, mask, radial_order=order, alpha_mode="fixed", alpha=0.01) < 1.1


@pytest.mark.parametrize("order", [4, 6])
def test_a_given_order_keeps_the_result(order):
    """The caller's voxel order (the previous fit's iteration counts) holds in the first pass."""
    import torch
    from cs_dmri_b200.autograd import DifferentiableShore
    ph, data, _ = tiled(15000)
    s = torch.from_numpy(np.ascontiguousarray(data.reshape(15000, -1), dtype=np.float32)).cuda()
    kw = dict(big_delta=ph.big_delta, small_delta=ph.small_delta, radial_order=order)
    by_index = DifferentiableShore(ph.bvals, ph.bvecs, schedule="index", **kw)
    by_count = DifferentiableShore(ph.bvals, ph.bvecs, schedule="previous", **kw)
    for alpha in (0.0005, 0.01):
        want = by_index.fit(s, alpha=alpha)
        for _ in range(2):
            assert torch.equal(by_count.fit(s, alpha=alpha), want)
