"""The warp-per-sample k-hop kernel where it can go wrong: fan-outs that do not divide a warp, hops just within and
beyond what a warp sorts in registers, rows too long for shared memory, fewer and more samples than warps."""
import numpy as np
import pytest

from conftest import kernel_constant, sm_count

pytestmark = pytest.mark.gpu
# resident warps of the GPU, by app
WARPS = {app: sm_count() * 8 * kernel_constant("nd_khop_rows.cu", name) for app, name in ((4, "CTAS"), (5, "CTAS_DISTINCT"))}


def _compare(nd, ndo, hg, app, fanout, S, seed=3, modes=(1, 2)):
    g = nd.Graph.from_csr(hg.row_ptr, hg.col, hg.w, hg.max_w)
    init = np.random.default_rng(S).integers(0, hg.V, S).astype(np.int32)
    init[::7] = hg.V
    s = nd.Sampler(g, nd.app_params(app, fanout=fanout, seed=seed), num_samples=S, first_sample=11, initial=init)
    exp = ndo.sample(hg, ndo.make_params(app, fanout=fanout, seed=seed), S, first=11, initial=init)
    for mode in modes:
        s.sample(mode)
        assert np.array_equal(s.final_samples(), exp["out"]), mode
        st = s.stats()
        assert st["sampled_edges"] == exp["counters"]["sampled_edges"] and st["live_pairs"] == exp["counters"]["live_pairs"]
        if app == 5:
            assert np.array_equal(s.aux()["hop_counts"], exp["hop_counts"])


@pytest.mark.parametrize("app", [4, 5])
@pytest.mark.parametrize("fanout", [[1], [32], [31, 2], [11, 3], [16, 16], [17, 15, 2], [32, 32], [2, 2, 2, 2, 2, 2, 2, 2], [1, 1, 32]])
def test_fanouts(nd, ndo, small_graph, app, fanout):
    _compare(nd, ndo, small_graph, app, fanout, 301, modes=(1, 2, 0))


@pytest.mark.parametrize("app", [4, 5])
@pytest.mark.parametrize("warps,more", [(0, 1), (0, 4), (0, 5), (1, -1), (1, 1), (16, 1), (17, 0)])
def test_sample_counts(nd, ndo, small_graph, app, warps, more):
    _compare(nd, ndo, small_graph, app, [3, 2], warps * WARPS[app] + more)


def test_rows_beyond_shared_memory(nd, ndo, small_graph):
    _compare(nd, ndo, small_graph, 4, [32, 32, 4], 40, modes=(1, 2))      # 5152 ids: the transit-parallel kernels
    _compare(nd, ndo, small_graph, 4, [31, 31, 3], 40, modes=(1, 2))      # 3875 ids: just below the limit
