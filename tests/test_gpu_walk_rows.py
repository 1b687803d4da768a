"""The lane-per-walk kernels (sample-parallel and load-balanced modes) where they can go wrong: rows that do not fill
the pieces they are written in, jobs just below and above the number of resident lanes, weights whose byte code
decides nothing, rows that shrink and grow between passes."""
import numpy as np
import pytest

from conftest import kernel_constant, sm_count

pytestmark = pytest.mark.gpu
# resident lanes of the GPU
LANES = sm_count() * kernel_constant("nd_walk_rows.cu", "ROWS_CTAS") * kernel_constant("nd_walk_rows.cu", "ROWS_THREADS")


def _graph(nd, hg):
    return nd.Graph.from_csr(hg.row_ptr, hg.col, hg.w, hg.max_w)


@pytest.mark.parametrize("app", [0, 1, 2, 3])
@pytest.mark.parametrize("steps", [1, 3, 7, 8, 9, 15, 16, 17, 24, 31, 100])
def test_row_pieces(nd, ndo, small_graph, app, steps):
    g = _graph(nd, small_graph)
    S = 1003
    rng = np.random.default_rng(steps)
    pr = nd.app_params(app, steps=steps, seed=7, stop_prob=0.1)
    s = nd.Sampler(g, pr, num_samples=S, first_sample=5)
    for mode in (1, 2, 0, 1):
        init = rng.integers(-1, small_graph.V, S).astype(np.int32)
        s.set_initial(init)
        s.sample(mode)
        clean = np.where(init < 0, small_graph.V, init).astype(np.int32)
        exp = ndo.sample(small_graph, ndo.make_params(app, steps=steps, seed=7, stop_prob=0.1), S, first=5, initial=clean)
        assert np.array_equal(s.final_samples(), exp["out"]), mode
        st = s.stats()
        assert all(st[k] == exp["counters"][k] for k in ("sampled_edges", "live_pairs", "weight_tries", "n2v_tries")), mode
        if mode == 1:
            live = s.live_pairs()
            n = (exp["out"] != small_graph.V).sum(axis=1)
            assert live[0] == (init >= 0).sum() and all(live[k] == (n >= k).sum() for k in range(1, steps))


@pytest.mark.parametrize("app", [0, 1, 2, 3])
@pytest.mark.parametrize("S", [1, 31, LANES, LANES + 1, LANES + 4097])
def test_job_sizes_around_the_resident_lanes(nd, ndo, small_graph, app, S):
    g = _graph(nd, small_graph)
    pr = nd.app_params(app, steps=5, seed=3, stop_prob=0.3)
    s = nd.Sampler(g, pr, num_samples=S)
    exp = ndo.sample(small_graph, ndo.make_params(app, steps=5, seed=3, stop_prob=0.3), S)
    for _ in range(2):
        s.sample(1)
        assert np.array_equal(s.final_samples(), exp["out"])
        assert s.stats()["live_pairs"] == exp["counters"]["live_pairs"]


@pytest.mark.parametrize("kind", ["equal", "tiny", "zero", "spread", "steps"])
def test_weights_at_the_edges_of_their_byte_code(nd, ndo, small_graph, kind):
    rng = np.random.default_rng(1)
    n = small_graph.E
    w = {"equal": np.full(n, 3.0), "tiny": rng.random(n) * 1e-42, "zero": np.where(rng.random(n) < 0.7, 0.0, 2.0),
         "spread": 10.0 ** rng.uniform(-6, 3, n), "steps": rng.integers(1, 257, n) / 256.0}[kind].astype(np.float32)
    src = np.repeat(np.arange(small_graph.V, dtype=np.int32), small_graph.degree())
    hg = ndo.csr_from_records(src, small_graph.col, w, V=small_graph.V)
    pr = nd.app_params(1, steps=12, seed=11)
    s = nd.Sampler(_graph(nd, hg), pr, num_samples=4000)
    s.sample(1)
    exp = ndo.sample(hg, ndo.make_params(1, steps=12, seed=11), 4000)
    assert np.array_equal(s.final_samples(), exp["out"])
    assert s.stats()["weight_tries"] == exp["counters"]["weight_tries"]


@pytest.mark.parametrize("app", [1, 2])
@pytest.mark.parametrize("kind", ["nan", "negative", "least", "below", "infinite"])
def test_maxima_that_rule_packed_weights_in_or_out(nd, ndo, small_graph, app, kind):
    """A caller's maxima: the packed weights decide by them, or the records do where they cannot."""
    rng = np.random.default_rng(2)
    n = small_graph.E
    w = (rng.random(n) + 0.25).astype(np.float32)
    odd = {"nan": np.nan, "negative": -1.0, "least": 2.0 ** -100, "below": 2.0 ** -101, "infinite": np.inf}[kind]
    mw = np.where(rng.random(small_graph.V) < 0.2, odd, small_graph.max_w).astype(np.float32)
    if kind == "infinite":   # a finite weight under an infinite maximum is never accepted
        w[rng.random(n) < 0.5] = np.inf
        src = np.repeat(np.arange(small_graph.V, dtype=np.int32), small_graph.degree())
        mw = np.zeros(small_graph.V, np.float32)
        np.maximum.at(mw, src, w)
    hg = ndo.HostGraph(small_graph.row_ptr, small_graph.col, w, mw)
    s = nd.Sampler(_graph(nd, hg), nd.app_params(app, steps=9, seed=4, stop_prob=0.1), num_samples=3000)
    s.sample(1)
    exp = ndo.sample(hg, ndo.make_params(app, steps=9, seed=4, stop_prob=0.1), 3000)
    assert np.array_equal(s.final_samples(), exp["out"])
    assert s.stats()["weight_tries"] == exp["counters"]["weight_tries"]


@pytest.mark.parametrize("V", [1 << 24, (1 << 24) + 1])
def test_ids_up_to_and_beyond_the_packed_width(nd, ndo, V):
    rng = np.random.default_rng(3)
    ids = np.unique(np.concatenate([rng.integers(0, V, 300), [0, V - 1, V - 2]])).astype(np.int32)
    src = np.concatenate([rng.choice(ids, 4000), [V - 1]]).astype(np.int32)
    dst = np.concatenate([rng.choice(ids, 4000), [V - 2]]).astype(np.int32)
    hg = ndo.csr_from_records(src, dst, (rng.random(len(src)) + 0.1).astype(np.float32), V=V)
    init = rng.choice(ids, 1000).astype(np.int32)
    for app in (1, 2):
        s = nd.Sampler(_graph(nd, hg), nd.app_params(app, steps=9, seed=4, stop_prob=0.1), num_samples=1000, initial=init)
        s.sample(1)
        exp = ndo.sample(hg, ndo.make_params(app, steps=9, seed=4, stop_prob=0.1), 1000, initial=init)
        assert np.array_equal(s.final_samples(), exp["out"]), app


@pytest.mark.parametrize("app", [1, 3])
@pytest.mark.parametrize("S", [2 * LANES, 2 * LANES + 33, 3 * LANES - 1])
def test_rounds_of_walks(nd, ndo, small_graph, app, S):
    rng = np.random.default_rng(S)
    able = np.flatnonzero(small_graph.degree() > 0)
    init = rng.choice(able, S).astype(np.int32)   # every walk can start: the list is as long as the job
    s = nd.Sampler(_graph(nd, small_graph), nd.app_params(app, steps=3, seed=3), num_samples=S, initial=init)
    exp = ndo.sample(small_graph, ndo.make_params(app, steps=3, seed=3), S, initial=init)
    for _ in range(2):
        s.sample(1)
        assert np.array_equal(s.final_samples(), exp["out"])
        assert s.stats()["live_pairs"] == exp["counters"]["live_pairs"]


@pytest.mark.parametrize("app", [0, 3])
@pytest.mark.parametrize("V,M", [(1 << 21, (1 << 23) - 1), (1 << 21, 1 << 23), (1 << 21, (1 << 23) + 1), (1 << 21, (1 << 23) + 2), ((1 << 21) + 1, 1 << 23),
                                 (3000, 1 << 23)])
def test_ids_of_21_bits(nd, app, V, M):
    """Against the exact-sort mode, which reads the plain ids."""
    g = nd.Graph.rmat(V, M, seed=3)
    init = np.random.default_rng(M).integers(0, V, 20000).astype(np.int32)
    s = nd.Sampler(g, nd.app_params(app, steps=15, seed=5), num_samples=len(init), initial=init)
    s.sample(0)
    exp = s.final_samples().copy()
    for mode in (1, 2):
        s.sample(mode)
        assert np.array_equal(s.final_samples(), exp), mode


@pytest.mark.parametrize("app", [0, 1, 2, 3])
@pytest.mark.parametrize("V,M", [(60_000, (1 << 21) - 3), (60_000, 1 << 21), (60_000, (1 << 21) + 1), ((1 << 22) - 1, 1 << 21), (1 << 22, (1 << 21) + 1)])
def test_entries_with_and_without_rows(nd, app, V, M):
    """Around 2^22 entries and 2^22 vertices, against the exact-sort mode, which reads the plain arrays."""
    g = nd.Graph.rmat(V, M, seed=3)
    init = np.random.default_rng(M).integers(0, V, 20000).astype(np.int32)
    s = nd.Sampler(g, nd.app_params(app, steps=15, seed=5, stop_prob=0.05), num_samples=len(init), initial=init)
    s.sample(0)
    exp = s.final_samples().copy()
    tries = s.stats()["weight_tries"]
    for mode in (1, 2):
        s.sample(mode)
        assert np.array_equal(s.final_samples(), exp) and s.stats()["weight_tries"] == tries, mode
