"""The choice of the FISTA kernel inside a CUDA graph: a warmed batch fit is
captured and replayed on other signals and another alpha, dense and sparse."""

import numpy as np
import pytest

from test_gpu_sparse import tiled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,v", [(6, 9000), (6, 12000), (4, 13000)])
@pytest.mark.parametrize("schedule", ["index", "previous"])
def test_replay_equals_the_eager_fit(order, v, schedule):
    import torch
    from cs_dmri_b200.autograd import DifferentiableShore
    ph, data, _ = tiled(v)
    rows = torch.from_numpy(np.ascontiguousarray(data.reshape(v, -1), dtype=np.float32)).cuda()
    kw = dict(big_delta=ph.big_delta, small_delta=ph.small_delta, radial_order=order, schedule=schedule)
    m = DifferentiableShore(ph.bvals, ph.bvecs, **kw)
    s, alpha = rows.clone(), torch.full((v,), 0.01, dtype=torch.float64, device="cuda")
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            m.fit(s, alpha)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = m.fit(s, alpha)
    eager = DifferentiableShore(ph.bvals, ph.bvecs, **{**kw, "schedule": "index"})
    for a, shift in ((0.01, 0), (0.0003, 7), (0.02, 20)):
        s.copy_(rows.roll(shift, 0))
        alpha.fill_(a)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, eager.fit(s, alpha))
    del graph
