"""Results and graphs through the staged copies: sizes around a piece and around the size below which the plain copy
is used, odd addresses, pinned destinations, several threads at once; the loader with weights that do not differ."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.mark.parametrize("nbytes", [4, 2 * MB - 4, 2 * MB, 2 * MB + 4, 9 * MB - 4, 9 * MB + 4, 41 * MB])
def test_final_samples_of_every_size(nd, small_graph, nbytes):
    import torch
    from nextdoor_b200 import dist as nd_dist
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    s = nd.Sampler(g, nd.app_params(0, steps=1, seed=2), num_samples=nbytes // 4)
    s.sample()
    exp = nd_dist.device_samples(s).cpu().numpy()
    assert np.array_equal(s.final_samples(), exp)
    raw = np.zeros(nbytes + 64, np.uint8)
    for off in (0, 4, 60):
        out = raw[off:off + nbytes].view(np.int32)
        out[:] = -9
        s.final_samples(out)
        assert np.array_equal(out, exp.reshape(-1))
    pinned = torch.full((nbytes // 4,), -9, dtype=torch.int32).pin_memory().numpy()
    s.final_samples(pinned)
    assert np.array_equal(pinned, exp.reshape(-1))


def test_several_threads_copy_at_once(nd, small_graph):
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    samplers = [nd.Sampler(g, nd.app_params(0, steps=10, seed=k), num_samples=300_000) for k in range(4)]
    for s in samplers:
        s.sample()
    exp = [s.final_samples() for s in samplers]
    wrong = []

    def work(k):
        for _ in range(5):
            if not np.array_equal(samplers[k].final_samples(), exp[k]):
                wrong.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("n", [0, 1, 2, 1000, 300_000])
@pytest.mark.parametrize("weights", ["same", "two", "low bits", "signs", "random"])
def test_loader_sorts_by_all_bits_that_differ(nd, ndo, n, weights):
    rng = np.random.default_rng(n)
    V = 700
    src, dst = rng.integers(0, V, n).astype(np.int32), rng.integers(0, V // 8, n).astype(np.int32)
    w = {"same": np.full(n, 1.5), "two": rng.choice([1.0, 1.0 + 2.0 ** -23], n), "low bits": 1.0 + rng.integers(0, 4, n) * 2.0 ** -22,
         "signs": rng.choice([-2.0, -1.0, 1.0, 2.0], n), "random": rng.random(n) * 4 + 1}[weights].astype(np.float32)
    g = nd.Graph.from_edge_records(src, dst, w)
    row_ptr, col, got_w, max_w = g.to_host()
    order = np.lexsort((w, dst, src))
    assert np.array_equal(col, dst[order]) and np.array_equal(got_w, w[order])
    assert np.array_equal(np.diff(row_ptr), np.bincount(src, minlength=g.V)[: g.V])
    exp_max = np.zeros(g.V, np.float32)
    np.maximum.at(exp_max, src, w)
    assert np.array_equal(max_w, exp_max)


@pytest.mark.parametrize("repeats", [2, 31, 32, 33, 34, 4095, 4096, 4097, 9000])
def test_loader_sorts_the_weights_of_repeated_edges(nd, repeats):
    rng = np.random.default_rng(repeats)
    pairs = np.stack([rng.integers(0, 40, 24), rng.integers(0, 40, 24)])
    e = rng.permutation(np.concatenate([np.repeat(np.arange(23), rng.integers(1, 40, 23)), np.full(repeats, 23)]))
    src, dst, w = pairs[0, e].astype(np.int32), pairs[1, e].astype(np.int32), (rng.random(len(e)) * 4 - 2).astype(np.float32)
    row_ptr, col, got_w, _ = nd.Graph.from_edge_records(src, dst, w).to_host()
    order = np.lexsort((w, dst, src))
    assert np.array_equal(col, dst[order]) and np.array_equal(got_w, w[order])


@pytest.mark.parametrize("S", [1, 31, 32, 255, 256, 257, 4095, 4097, 9000])
@pytest.mark.parametrize("stop", [0.02, 0.6])
def test_rows_packed_at_the_edges_of_a_chunk(nd, small_graph, S, stop):
    import torch
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    V, steps = small_graph.V, 100
    s = nd.Sampler(g, nd.app_params(2, steps=steps, seed=5, stop_prob=stop), num_samples=S)
    full = torch.full((S, steps), V, dtype=torch.int32, device="cuda")
    full_len = torch.zeros(S, dtype=torch.int32, device="cuda")
    scratch = torch.empty(nd.rows_scratch_words(S), dtype=torch.int32, device="cuda")
    host, host_len = np.full(S * steps, V, np.int32), np.zeros(S, np.int32)
    rng = np.random.default_rng(S)
    for _ in range(3):
        s.set_initial(np.where(rng.random(S) < 0.2, -1, rng.integers(0, V, S)).astype(np.int32))
        s.sample(1)
        dense = s.final_samples()
        len_ptr, vals_ptr = s.pack_rows()
        assert s.pack_rows_total() == int((dense != V).sum())
        nd.rows_unpack(0, None, S, steps, V, len_ptr, vals_ptr, full.data_ptr(), full_len.data_ptr(), scratch.data_ptr())
        torch.cuda.synchronize()
        assert np.array_equal(full.cpu().numpy(), dense)
        s.host_update_begin(host, host_len)
        s.host_update_fetch()
        s.host_update_finish()
        assert np.array_equal(host.reshape(S, steps), dense) and np.array_equal(host_len, (dense != V).sum(axis=1))


@pytest.mark.parametrize("call", ["host_update_begin", "host_update_fetch", "host_update_finish"])
@pytest.mark.parametrize("depth", [1, 2])
def test_a_pipeline_goes_on_after_an_error(nd, small_graph, monkeypatch, call, depth):
    import torch
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    S, steps = 9001, 30
    streams = torch.cuda.Stream(), torch.cuda.Stream()
    params = nd.app_params(2, steps=steps, seed=5, stop_prob=0.2)
    pipe = nd.PipelinedSampler(g, params, S, chunks=3, depth=depth, sparse_rows=True, stream=streams[0].cuda_stream,
                               copy_stream=streams[1].cuda_stream)
    seeds = [np.random.default_rng(k).integers(0, g.V, S).astype(np.int32) for k in range(2)]
    outs = [np.zeros(S * steps, np.int32) for _ in range(2)]
    pipe.run(seeds[0], outs[0])

    def failing(smp):
        def fails(*args):
            if call == "host_update_finish":      # the update is over all the same
                type(smp).host_update_finish(smp)
            raise nd.NdError(2, "no")
        return fails

    with monkeypatch.context() as m:
        for parts in pipe.sets:
            m.setattr(parts[1][2], call, failing(parts[1][2]))
        with pytest.raises(nd.NdError):
            for k in (0, 1):
                pipe.run_async(seeds[1 - k], outs[k])
            pipe.wait()
    for k in (0, 1, 1):
        pipe.run_async(seeds[k], outs[k])
    pipe.wait()
    for k in (0, 1):
        s = nd.Sampler(g, params, num_samples=S, initial=seeds[k])
        s.sample()
        assert np.array_equal(outs[k].reshape(S, steps), s.final_samples())


@pytest.mark.parametrize("app", [6, 8, 9])
@pytest.mark.parametrize("L,B,S", [(48, 50, 70), (7, 5, 2675), (1, 3, 43_691), (64, 64, 33)])
def test_adjacency_crosses_as_bits(nd, ndo, small_graph, app, L, B, S):
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    s = nd.Sampler(g, nd.app_params(app, steps=2, fanout=L, batch=B, seed=6), num_samples=S)
    s.sample()
    exp = ndo.sample(small_graph, ndo.make_params(app, steps=2, fanout=L, batch=B, seed=6), S)
    same = (s.final_samples() == exp["out"]).all(axis=1)
    # LADIES: a draw on the edge of an interval may fall to its neighbour.  The oracle adds a candidate's terms up in 32
    # bits, each sum off by up to 6e-8 of itself, so that the edges lie about 1e-6 of the whole apart in all: of the
    # S * 2 * L draws (at most 87,382) 0.1 is expected to differ
    assert (~same).sum() <= (1 if app == 9 else 0)
    aux = s.aux()
    for k in ("adj_row", "adj_col"):
        assert np.array_equal(aux[k].reshape(S, -1)[same], exp[k].reshape(S, -1)[same])
    assert (aux["adj_row"] >= 0).sum() > 0


@pytest.mark.parametrize("L,B,S", [(33, 20, 3), (33, 20, 300), (64, 64, 100)])
def test_one_array_of_an_adjacency(nd, small_graph, L, B, S):
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    s = nd.Sampler(g, nd.app_params(6, steps=3, fanout=L, batch=B, seed=6), num_samples=S)
    s.sample()
    both = s.aux()
    for k in ("adj_row", "adj_col"):
        one = np.full(both[k].size + 1, 7, np.int32)
        ptr = one.ctypes.data
        nd.check(nd.lib.nd_sampler_aux(s._h, ptr if k == "adj_row" else None, ptr if k == "adj_col" else None, None, None))
        assert np.array_equal(one[:-1], both[k].reshape(-1)) and one[-1] == 7


def test_results_own_their_memory(nd, small_graph):
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    s = nd.Sampler(g, nd.app_params(0, steps=10, seed=2), num_samples=300_000)
    s.sample()
    exp = np.zeros(3_000_000, np.int32)
    s.final_samples(exp)
    kept = [s.final_samples() for _ in range(3)]
    for a in kept:
        a[:] = -5
    row = kept[1][7]                     # a view holds the whole
    del kept[1]
    for _ in range(5):                   # new memory, then lent again, then pinned
        assert np.array_equal(s.final_samples().reshape(-1), exp)
    assert (row == -5).all() and (kept[0] == -5).all() and (kept[1] == -5).all()
    last = s.final_samples()
    del s, g
    assert np.array_equal(last.reshape(-1), exp)   # results outlive the sampler


@pytest.mark.parametrize("n,V,weights,repeats", [((1 << 21) - 1, 50_000, "random", 0), (1 << 21, 50_000, "random", 3000), ((1 << 21) + 33, 1 << 20, "same", 0),
                                                 ((1 << 21) + 33, 3000, "signs", 9000)])
def test_loader_of_ids_before_weights(nd, n, V, weights, repeats):
    """Sizes from which on the ids are sorted while the weights are on their way: the same CSR, whatever repeats."""
    rng = np.random.default_rng(n + V)
    src, dst = rng.integers(0, V, n).astype(np.int32), (V * rng.random(n) ** 4).astype(np.int32)
    src[:repeats], dst[:repeats] = 7, 11
    w = {"random": rng.random(n) * 4 + 1, "same": np.full(n, 2.5), "signs": rng.choice([-2.0, -1.0, 1.0, 2.0], n)}[weights].astype(np.float32)
    at = rng.permutation(n)
    src, dst, w = src[at], dst[at], w[at]
    g = nd.Graph.from_edge_records(src, dst, w)
    row_ptr, col, got_w, max_w = g.to_host()
    order = np.lexsort((w, dst, src))
    assert g.V == max(src.max(), dst.max()) + 1 and g.max_degree == np.bincount(src).max()
    assert np.array_equal(col, dst[order]) and np.array_equal(got_w, w[order])
    assert np.array_equal(np.diff(row_ptr), np.bincount(src, minlength=g.V))
    exp_max = np.zeros(g.V, np.float32)
    np.maximum.at(exp_max, src, w)
    assert np.array_equal(max_w, exp_max)
    dst[n // 2] = -3
    with pytest.raises(nd.NdError):
        nd.Graph.from_edge_records(src, dst, w)
    dst[n // 2] = 3
    assert nd.Graph.from_edge_records(src, dst, w).E == n


@pytest.mark.parametrize("nbytes", [(256 << 10) - 4, 256 << 10, (256 << 10) + 4])
def test_results_of_the_smallest_size_that_is_kept(nd, small_graph, nbytes):
    """New memory, lent again, pinned: every result is the job's, and one that a caller holds stays as it is."""
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    jobs = [nd.Sampler(g, nd.app_params(0, steps=1, seed=seed), num_samples=nbytes // 4) for seed in (2, 3)]
    exp = []
    for s in jobs:
        s.sample()
        out = np.full(nbytes // 4, -9, np.int32)
        s.final_samples(out)
        exp.append(out.reshape(-1, 1))
    held = jobs[0].final_samples()
    for _ in range(4):
        for s, e in zip(jobs, exp):
            assert np.array_equal(s.final_samples(), e)
    assert np.array_equal(held, exp[0]) and not np.array_equal(exp[0], exp[1])


def test_small_results_leave_the_large_ones_their_memory(nd):
    """A queue of results below 2 MB, held and dropped again and again, and a large one that is lent, pinned, kept."""
    import torch
    large = nd.Sampler(nd.Graph.rmat(5000, 40_000, seed=1), nd.app_params(0, steps=100, seed=1), num_samples=50_000)
    small = nd.Sampler(large.graph, nd.app_params(0, steps=1, seed=2), num_samples=1 << 16)
    large.sample()
    small.sample()
    exp_large, exp = np.zeros((50_000, 100), np.int32), np.zeros((1 << 16, 1), np.int32)
    large.final_samples(exp_large)
    small.final_samples(exp)
    for _ in range(3):
        queue = [small.final_samples() for _ in range(300)]
        assert all(np.array_equal(a, exp) for a in queue)
        del queue
    for turn in range(3):
        result = large.final_samples()
        assert np.array_equal(result, exp_large)
        assert turn == 0 or torch.from_numpy(result).is_pinned()
        del result
    at = large.final_samples().ctypes.data
    queue = [small.final_samples() for _ in range(300)]
    del queue
    result = large.final_samples()
    assert result.ctypes.data == at and torch.from_numpy(result).is_pinned() and np.array_equal(result, exp_large)
