"""Calls that fail for want of device memory: what they leave behind."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("app", [0, 3, 4, 9])
def test_a_failed_call_does_not_fail_the_next(nd, small_graph, app):
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    pr = nd.app_params(app, seed=1)
    s = nd.Sampler(g, pr, num_samples=50)
    s.sample()
    expected = s.final_samples().copy()
    for _ in range(2):
        with pytest.raises(nd.NdError, match="memory"):
            nd.Sampler(g, nd.app_params(1, steps=200, seed=1), num_samples=1 << 30)   # 858 GB of rows
        s = nd.Sampler(g, pr, num_samples=50)
        s.sample()
        assert np.array_equal(s.final_samples(), expected)
