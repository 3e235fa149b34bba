"""The device fit is ordered with the work queued before it on the caller's
current stream, torch's default stream (handle 0) included."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", ["default", "default-given", "side"])
@pytest.mark.parametrize("dtype", ["bool", "uint8"])
def test_the_fit_waits_for_its_inputs(where, dtype):
    import torch
    from cs_dmri_b200 import shore_fit_device
    from cs_dmri_b200.phantom import make_phantom
    ph = make_phantom((6, 6, 3), seed=3)
    ready = torch.from_numpy(np.ascontiguousarray(ph.data)).cuda()
    keep = torch.ones((6, 6, 3), dtype=getattr(torch, dtype), device="cuda")
    kw = dict(big_delta=ph.big_delta, small_delta=ph.small_delta, alpha_mode="fixed", alpha=0.01)
    torch.cuda.synchronize()
    want, _ = shore_fit_device(ready, keep, ph.bvals, ph.bvecs, **kw)
    torch.cuda.synchronize()
    assert bool(want.any())
    stream = torch.cuda.Stream() if where == "side" else torch.cuda.default_stream()
    late, mask = torch.zeros_like(ready), torch.zeros_like(keep)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(100_000_000)  # about 50 ms: the copies below are still queued when the fit is called
        late.copy_(ready)
        mask.copy_(keep)
        got, _ = shore_fit_device(late, mask, ph.bvals, ph.bvecs, stream=stream if where == "default-given" else None,
                                  **kw)
        twice = 2.0 * got  # and work queued after it reads its result
    torch.cuda.synchronize()
    assert torch.equal(got, want) and torch.equal(twice, 2.0 * want)
