"""Importance layers where the degrees do not fit the packed codes: vertices around the degrees at which the second byte
and the list of big vertices begin, vertices without neighbours among the candidates, graphs that end inside a group."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [6000, 6144, 20_001])
@pytest.mark.parametrize("degrees", [(1, 2), (255, 256, 257), (2046, 2047), (2047, 2048, 2049, 5000)])
@pytest.mark.parametrize("scratch", ["0", "1"])
def test_fastgcn_weights_at_the_edges_of_the_codes(nd, ndo, monkeypatch, V, degrees, scratch):
    monkeypatch.setenv("ND_COLLECTIVE_SORT", "0")
    monkeypatch.setenv("ND_COLLECTIVE_BITMAP_GLOBAL", scratch)
    rng = np.random.default_rng(V + degrees[0])
    hubs = np.unique(np.concatenate([rng.integers(0, 40, 20), rng.integers(0, V, 40), [V - 1]]))
    deg = np.where(rng.random(V) < 0.1, 0, rng.integers(1, 6, V))
    deg[hubs] = rng.choice(degrees, len(hubs))
    src = np.repeat(np.arange(V), deg).astype(np.int32)
    dst = np.where(rng.random(len(src)) < 0.2, rng.choice(hubs, len(src)), rng.integers(0, V, len(src))).astype(np.int32)
    hg = ndo.csr_from_records(src, dst, np.ones(len(src), np.float32), V=V)
    g = nd.Graph.from_csr(hg.row_ptr, hg.col, hg.w, hg.max_w)
    S, L = 60, 32
    s = nd.Sampler(g, nd.app_params(8, steps=2, fanout=L, batch=24, seed=3), num_samples=S, first_sample=2)
    s.sample()
    exp = ndo.sample(hg, ndo.make_params(8, steps=2, fanout=L, batch=24, seed=3), S, first=2)
    aux = s.aux()
    assert np.array_equal(s.final_samples(), exp["out"])   # whole numbers: the sums are exact
    assert np.array_equal(aux["prob"].reshape(-1), exp["prob"].reshape(-1))
    assert np.array_equal(aux["adj_row"], exp["adj_row"]) and np.array_equal(aux["adj_col"], exp["adj_col"])


@pytest.mark.parametrize("app", [8, 9])
@pytest.mark.parametrize("created,sampled", [("0", "1"), ("1", "0")])
def test_a_sampler_keeps_the_layout_it_was_created_with(nd, monkeypatch, small_graph, app, created, sampled):
    """The switch that moves the bitmaps to global scratch is asked when the buffers are sized, not again by a job."""
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    out = []
    for at_creation in (created, sampled):
        monkeypatch.setenv("ND_COLLECTIVE_BITMAP_GLOBAL", at_creation)
        s = nd.Sampler(g, nd.app_params(app, steps=2, fanout=32, batch=24, seed=3), num_samples=400)
        monkeypatch.setenv("ND_COLLECTIVE_BITMAP_GLOBAL", sampled)
        s.sample()
        out.append(s.final_samples())
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("app,sizes", [(8, [(16, 16), (600, 600)]), (9, [(16, 16), (600, 600)]), (7, [(560, 560), (640, 640)]), (4, [(16, 15, 13), (15, 15, 17)])])
def test_threads_with_different_shared_memory(nd, small_graph, app, sizes):
    """The limit of a kernel's dynamic shared memory is the kernel's: a thread that launches with little must not lower
    it under another's launch."""
    import threading
    wide = nd.Graph.rmat(300_000, 600_000, seed=1)
    graphs = [nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w), wide]
    samplers = []
    for g, size in zip(graphs, sizes):
        pr = nd.app_params(app, fanout=list(size), seed=3) if app == 4 else nd.app_params(app, steps=1, fanout=size[0], batch=size[1], seed=3)
        samplers.append(nd.Sampler(g, pr, num_samples=2))
    errors = []

    def work(s):
        try:
            for _ in range(300 if app == 7 else 1500):
                s.sample(sync=False)
            s.sync()
        except nd.NdError as e:
            errors.append(str(e))

    threads = [threading.Thread(target=work, args=(s,)) for s in samplers]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("kind,hubs", [("apart", 1023), ("apart", 1025), ("apart", 2500), ("equal", 1500), ("few ties", 1500)])
@pytest.mark.parametrize("app", [8, 9])
def test_bitmaps_go_to_the_vertices_with_the_most_neighbours(nd, ndo, app, kind, hubs):
    """1024 neighbourhoods are kept as bitmaps; of more vertices with enough neighbours the largest have one, of equal
    ones those with the lowest ids."""
    import ctypes as C
    import torch
    V = 8000                                       # 256 neighbours and more
    rng = np.random.default_rng(hubs)
    ids = rng.permutation(V)[:hubs]
    deg = np.zeros(V, np.int64)
    deg[rng.integers(0, V, 2000)] = rng.integers(1, 250, 2000)
    deg[ids] = {"apart": 256 + np.arange(hubs) // 2, "equal": np.full(hubs, 300), "few ties": 256 + rng.integers(0, 4, hubs)}[kind]
    src = np.repeat(np.arange(V), deg).astype(np.int32)
    dst = np.concatenate([(v + 1 + np.arange(d) * 13) % V for v, d in enumerate(deg) if d]).astype(np.int32)
    hg = ndo.csr_from_records(src, dst, np.ones(len(src), np.float32), V=V)
    g = nd.Graph.from_csr(hg.row_ptr, hg.col, hg.w, hg.max_w)
    s = nd.Sampler(g, nd.app_params(app, steps=2, fanout=32, batch=24, seed=3), num_samples=80)
    p = C.c_void_p()
    nd.check(nd.lib.nd_graph_hub_slots(g._h, C.byref(p)))
    shape = {"shape": (V,), "typestr": "<i4", "data": (p.value, False), "version": 3}
    slot = torch.as_tensor(type("Slots", (), {"__cuda_array_interface__": shape})(), device="cuda").cpu().numpy()
    order = np.lexsort((np.arange(V), -deg))
    with_bitmap = order[:1024][deg[order[:1024]] >= 256]
    assert np.array_equal(np.flatnonzero(slot >= 0), np.sort(with_bitmap))
    assert np.array_equal(np.sort(slot[slot >= 0]), np.arange(len(with_bitmap)))
    s.sample()
    exp = ndo.sample(hg, ndo.make_params(app, steps=2, fanout=32, batch=24, seed=3), 80)
    assert np.array_equal(s.final_samples(), exp["out"])


@pytest.mark.parametrize("steps", [23, 24, 25, 4_098_254])
def test_reference_layers_of_many_steps(nd, ndo, small_graph, steps):
    """The bytes of the last one's layers, all in one pass, are 2904 beyond 2^32."""
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    s = nd.Sampler(g, nd.app_params(6, steps=steps, fanout=1, batch=1, seed=3), num_samples=1)
    s.sample()
    exp = ndo.sample(small_graph, ndo.make_params(6, steps=steps, fanout=1, batch=1, seed=3), 1)
    aux = s.aux()
    assert np.array_equal(s.final_samples(), exp["out"])
    assert np.array_equal(aux["adj_row"], exp["adj_row"]) and np.array_equal(aux["adj_col"], exp["adj_col"])


@pytest.mark.parametrize("V,M,B,L", [(2000, 12_000, 24, 32), (60_000, 3_000_000, 500, 64)])
@pytest.mark.parametrize("scratch", ["0", "1"])
@pytest.mark.parametrize("app", [8, 9])
def test_rows_in_any_order(nd, monkeypatch, app, scratch, V, M, B, L):
    """CSR arrays of a caller whose rows do not ascend have the layers of the same graph with rows that do."""
    monkeypatch.setenv("ND_COLLECTIVE_BITMAP_GLOBAL", scratch)
    row_ptr, col, w, max_w = nd.Graph.rmat(V, M, seed=1).to_host()
    rng = np.random.default_rng(V)
    order = np.lexsort((rng.random(len(col)), np.repeat(np.arange(V), np.diff(row_ptr))))
    init = rng.integers(0, V, 40 * B).astype(np.int32)
    out = []
    for c, x in ((col, w), (col[order], w[order])):
        s = nd.Sampler(nd.Graph.from_csr(row_ptr, c, x, max_w), nd.app_params(app, steps=2, fanout=L, batch=B, seed=3), num_samples=40, initial=init)
        s.sample()
        out.append((s.final_samples(), s.aux()["prob"], s.stats()["union_unique"]))
    assert V < 16_384 or out[0][2] / 80 > 16_384        # more candidates than an accumulator tile holds
    # the row sums are added up in another order, to 1e-16: less than one draw in 10^9 can fall to its neighbour for it
    assert np.array_equal(out[0][0], out[1][0]) and out[0][2] == out[1][2]
    assert np.allclose(out[0][1], out[1][1], rtol=1e-6, atol=0)


def _ladies(nd, ndo, hg, S, B, L, init, adjacency=True):
    """Against 64-bit sums of the 32-bit terms.  2^18 terms added up in any order differ by 2^18 * 2^-53 of the total at
    most: a draw may fall to another candidate only that near to the end of one."""
    V, steps = hg.V, 2
    s = nd.Sampler(nd.Graph.from_csr(hg.row_ptr, hg.col, hg.w, hg.max_w), nd.app_params(9, steps=steps, fanout=L, batch=B, seed=3), num_samples=S, initial=init)
    s.sample()
    got, aux = s.final_samples().reshape(S, steps, L), s.aux()
    prob, seen = aux["prob"].reshape(S, steps, L), 0
    for smp in range(S):
        for step in range(steps):
            transits = init.reshape(S, B)[smp] if step == 0 else got[smp, step - 1]
            transits = transits[transits < V]
            rows = [slice(hg.row_ptr[t], hg.row_ptr[t + 1]) for t in transits]
            ids = np.concatenate([hg.col[r] for r in rows] or [np.zeros(0, np.int32)])
            share = np.concatenate([hg.w[r] / np.float32(hg.w[r].astype(np.float64).sum()) for r in rows] or [np.zeros(0, np.float32)])
            cand, at = np.unique(ids, return_inverse=True)
            seen += len(cand)
            if len(cand) == 0:
                assert (got[smp, step] == V).all()
                continue
            cdf = np.cumsum(np.bincount(at, (share * share).astype(np.float64)))
            u = np.array([ndo.lib().ndo_uniform(3, smp, step, j, 0) for j in range(L)], np.float32)
            target = u.astype(np.float64) * cdf[-1]
            mine = np.minimum(np.searchsorted(cand, got[smp, step]), len(cand) - 1)
            assert np.array_equal(cand[mine], got[smp, step])
            bound = 2.0 ** -35 * cdf[-1]
            before = np.concatenate([[0.0], cdf])[mine]
            assert (cdf[mine] >= target - bound).all() and (before <= target + bound).all()
            assert (prob[smp, step] > 0).all()
            assert np.allclose(prob[smp, step], (cdf[mine] - before) / cdf[-1], rtol=1e-6, atol=2.0 ** -35)
    assert s.stats()["union_unique"] == seen
    if adjacency:   # (whose probes ask for lists that ascend)
        assert ndo.check_adjacency(hg, ndo.make_params(9, steps=steps, fanout=L, batch=B, seed=3), S, init, s.final_samples(), aux["adj_row"], aux["adj_col"]) == 0


@pytest.mark.parametrize("V,B,L", [(129, 3, 1), (200_000, 100, 300), (200_000, 40, 31), (1_100_000, 64, 33), (1_300_000, 64, 64)])
def test_ladies_groups_and_accumulators(nd, ndo, V, B, L):
    """More groups drawn from than have accumulators at a time, groups that end behind the last vertex, lists that begin and end
    anywhere in an oct, the bitmap's place with and without room for them."""
    hg = ndo.rmat_graph(V, max(8 * V, 600) if V < 500_000 else 3 * V, seed=2)
    init = np.random.default_rng(V + L).integers(0, V, 20 * B).astype(np.int32)
    _ladies(nd, ndo, hg, 20, B, L, init)


@pytest.mark.parametrize("V", [3_000_000, 9_000_000, 20_000_000])
def test_ladies_of_many_vertices(nd, ndo, V):
    """Larger groups, then their sums in global scratch."""
    rng = np.random.default_rng(V)
    ids = rng.integers(0, V, 3000)
    src = np.concatenate([rng.choice(ids, 60_000), [V - 1]]).astype(np.int32)
    dst = np.concatenate([rng.choice(ids, 60_000), [ids[0]]]).astype(np.int32)
    hg = ndo.csr_from_records(src, dst, (rng.random(len(src)) + 0.1).astype(np.float32), V=V)
    _ladies(nd, ndo, hg, 6, 32, 64, rng.choice(ids, 6 * 32).astype(np.int32))


# draw 44 of this sample is 0xffffffd3 with seed 0: the one in 2^25 that the uniform number 1.0 comes from
TOP_SAMPLE, TOP_SLOT = 571_925, 44


def _top_layer(nd, ndo, V, ids, w, L=64):
    """The layer of a batch that is vertex 0 alone, whose neighbours are `ids`."""
    assert ndo.lib().ndo_uniform(0, TOP_SAMPLE, 0, TOP_SLOT, 0) == 1.0
    src, order = np.zeros(len(ids), np.int32), np.argsort(ids, kind="stable")
    hg = ndo.csr_from_records(src, ids[order].astype(np.int32), w[order].astype(np.float32), V=V)
    s = nd.Sampler(nd.Graph.from_csr(hg.row_ptr, hg.col, hg.w, hg.max_w), nd.app_params(9, steps=1, fanout=L, batch=1, seed=0), num_samples=1,
                   first_sample=TOP_SAMPLE, initial=np.zeros(1, np.int32))
    s.sample()
    return s.final_samples()[0], s.aux()["prob"]


@pytest.mark.parametrize("V", [3600, 70_000, 200_000, 1_300_000])
@pytest.mark.parametrize("scratch", ["0", "1"])
def test_ladies_draws_end_where_there_are_candidates(nd, ndo, monkeypatch, V, scratch):
    """Weights over eight decades, with which the sums of the groups are not exact, one neighbour in a group, and most groups
    without any, those behind the last one among them."""
    monkeypatch.setenv("ND_COLLECTIVE_BITMAP_GLOBAL", scratch)
    for seed in range(5, 25):
        rng = np.random.default_rng(seed)
        n = 22 if V == 3600 else int(rng.integers(20, 300))
        ids = 128 * rng.permutation(V // 128 - 2)[:n]
        w = 10 ** rng.uniform(-8, 0, n)
        if V == 3600:
            ids = np.sort(ids)
        layer, prob = _top_layer(nd, ndo, V, ids, w)
        assert np.isin(layer, ids).all(), (seed, layer[~np.isin(layer, ids)])
        assert (prob > 0).all(), seed


@pytest.mark.parametrize("V", [3600, 200_000])
@pytest.mark.parametrize("sort", ["0", "1"])
def test_ladies_draws_no_neighbour_of_weight_zero(nd, ndo, monkeypatch, V, sort):
    """Groups of a dozen candidates with weights over eight decades, between and behind them neighbours that cannot be drawn."""
    monkeypatch.setenv("ND_COLLECTIVE_SORT", sort)
    for seed in range(190):
        rng = np.random.default_rng(seed)
        ids = np.sort((128 * rng.permutation(V // 128 - 2)[:8, None] + rng.permutation(60)[:12]).reshape(-1))
        w = 10 ** rng.uniform(-8, 0, len(ids))
        nothing = np.setdiff1d(np.concatenate([ids + 1, ids + 40]), ids)
        layer, prob = _top_layer(nd, ndo, V, np.concatenate([ids, nothing]), np.concatenate([w, np.zeros(len(nothing))]))
        assert np.isin(layer, ids).all(), (seed, layer[~np.isin(layer, ids)])
        assert (prob > 0).all(), seed


@pytest.mark.parametrize("order,decades", [("ascending", 0), ("ascending", 8), ("hub's list", 0)])
@pytest.mark.parametrize("repeats", [1, 40])
def test_ladies_hubs_by_tables(nd, ndo, order, decades, repeats):
    """Hubs whose neighbours occur once and many times, whose lists end inside a group, and one whose list is in another order;
    weights of one size and over eight decades."""
    V, rng = 40_000, np.random.default_rng(repeats)
    hubs = np.array([0, 5, 127, 128, 20_000, V - 1])
    deg = rng.integers(0, 9, V)
    deg[hubs] = [300, 312, 313, 5000, 9001, 30_000]     # V / 128 = 312: one of them is none
    src = np.repeat(np.arange(V), deg).astype(np.int32)
    dst = (V * rng.random(len(src)) ** 2).astype(np.int32)
    often = np.isin(src, hubs) & (rng.random(len(src)) < 0.5)
    dst[often] = dst[often] // repeats * repeats        # on average `repeats` times the same neighbour
    toward = ~np.isin(src, hubs) & (rng.random(len(src)) < 0.3)
    dst[toward] = rng.choice(hubs, toward.sum())
    w = 10 ** rng.uniform(-decades, 0, len(src)) if decades else rng.random(len(src)) + 0.1
    hg = ndo.csr_from_records(src, dst, w.astype(np.float32), V=V)
    if order != "ascending":
        a, b = hg.row_ptr[20_000], hg.row_ptr[20_001]
        hg.col[a:b], hg.w[a:b] = hg.col[a:b][::-1].copy(), hg.w[a:b][::-1].copy()
    init = np.where(rng.random(30 * 24) < 0.2, rng.choice(hubs, 30 * 24), rng.integers(0, V, 30 * 24)).astype(np.int32)
    _ladies(nd, ndo, hg, 30, 24, 48, init, adjacency=order == "ascending")


@pytest.mark.parametrize("V,share,largest,batch", [(20_001, 0.05, 300, 24), (6144, 0.2, 2047, 24), (20_001, 0.02, 300, 24), (70_000, 0.0, 5000, 4),
                                                   (70_000, 0.001, 9000, 300), (6000, 0.0, 1 << 22, 24), (50_000, 0.0, (1 << 22) + 9, 6)])
@pytest.mark.parametrize("scratch", ["0", "1"])
def test_fastgcn_weights_of_listed_vertices(nd, ndo, monkeypatch, V, share, largest, batch, scratch):
    """A byte per degree or two, by the share of the vertices that do not fit one; few and many entries beside the hubs';
    squares that are not whole in 24 bits, and weights that the sums of the groups do not hold (from 2^22 neighbours)."""
    monkeypatch.setenv("ND_COLLECTIVE_BITMAP_GLOBAL", scratch)
    rng = np.random.default_rng(V + largest)
    deg = np.where(rng.random(V) < 0.1, 0, rng.integers(1, 6, V))
    many = rng.random(V) < share
    deg[many] = rng.integers(256, largest, many.sum()) if share else 0
    top = rng.choice(V, 6, replace=False)
    deg[top] = [largest, largest - 1, largest // 2, 4097, 256, 255]
    src = np.repeat(np.arange(V), deg).astype(np.int32)
    dst = np.where(rng.random(len(src)) < 0.2, rng.choice(top, len(src)), rng.integers(0, V, len(src))).astype(np.int32)
    hg = ndo.csr_from_records(src, dst, np.ones(len(src), np.float32), V=V)
    S, L, steps = 40, 32, 2 if largest < 1 << 20 else 1
    initial = rng.integers(0, V, S * batch).astype(np.int32)
    if steps == 1:
        initial[deg[initial] > 2] = int(np.argmax(deg == 2))   # (lists of millions take the oracle long)
    s = nd.Sampler(nd.Graph.from_csr(hg.row_ptr, hg.col, hg.w, hg.max_w), nd.app_params(8, steps=steps, fanout=L, batch=batch, seed=3), num_samples=S, initial=initial)
    s.sample()
    exp = ndo.sample(hg, ndo.make_params(8, steps=steps, fanout=L, batch=batch, seed=3), S, initial=initial)
    aux = s.aux()
    assert np.array_equal(s.final_samples(), exp["out"])   # whole numbers below 2^53: the sums are exact
    assert np.array_equal(aux["prob"].reshape(-1), exp["prob"].reshape(-1))
    assert np.array_equal(aux["adj_row"], exp["adj_row"]) and np.array_equal(aux["adj_col"], exp["adj_col"])
    assert s.stats()["union_unique"] == exp["counters"]["union_unique"]


@pytest.mark.parametrize("V,B,L", [(3000, 24, 33), (70_000, 64, 64)])
@pytest.mark.parametrize("app", [8, 9])
def test_layers_by_number_of_samples(nd, app, V, B, L):
    """One to four samples share an SM by how many there are (148 SMs); a sample's layers do not depend on it."""
    g = nd.Graph.rmat(V, 10 * V, seed=1)
    init = np.random.default_rng(V).integers(0, V, 600 * B).astype(np.int32)

    def job(first, S):
        s = nd.Sampler(g, nd.app_params(app, steps=2, fanout=L, batch=B, seed=3), num_samples=S, first_sample=first, initial=init[first * B:(first + S) * B])
        s.sample()
        aux = s.aux()
        return [x.reshape(S, -1) for x in (s.final_samples(), aux["adj_row"], aux["adj_col"], aux["prob"])]

    one = [np.concatenate(x) for x in zip(*(job(first, 120) for first in range(0, 600, 120)))]
    for first, S in [(0, 600), (600 - 148, 148), (7, 149), (150, 296), (0, 312), (3, 444), (100, 445)]:
        for got, exp in zip(job(first, S)[:3], one):
            assert np.array_equal(got, exp[first:first + S])
        assert np.allclose(job(first, S)[3], one[3][first:first + S], rtol=1e-6, atol=0)   # 32-bit results of 64-bit sums in another order


@pytest.mark.parametrize("app,B,L", [(8, 40, 1), (8, 40, 32), (9, 70, 33), (9, 70, 64), (8, 70, 65), (9, 40, 100), (8, 40, 129), (9, 70, 300)])
def test_adjacency_by_length_of_the_lists(nd, ndo, app, B, L):
    """Lists around the 32 parts in which they are looked through, none, short, with repeated edges; hubs (V / 128 neighbours)."""
    V = 40_000
    rng = np.random.default_rng(L)
    deg = rng.choice([0, 1, 2, 3, 31, 32, 33, 63, 64, 65, 95, 97, 255, 311, 312, 313, 900], V, p=[.3, .1, .1, .1, .05, .05, .05] + [.025] * 9 + [.025])
    src = np.repeat(np.arange(V), deg).astype(np.int32)
    dst = np.where(rng.random(len(src)) < 0.5, rng.integers(0, 60, len(src)) * 661, rng.integers(0, V, len(src))).astype(np.int32)   # (the 60 are drawn again and again)
    hg = ndo.csr_from_records(src, dst, np.ones(len(src), np.float32), V=V)
    g = nd.Graph.from_csr(hg.row_ptr, hg.col, hg.w, hg.max_w)
    S, steps = 30, 2
    init = rng.integers(0, V, S * B).astype(np.int32)
    s = nd.Sampler(g, nd.app_params(app, steps=steps, fanout=L, batch=B, seed=3), num_samples=S, initial=init)
    s.sample()
    out, aux = s.final_samples().reshape(S, steps, L), s.aux()
    rows, found = aux["adj_row"].reshape(S, steps, -1), 0
    for k in range(S):
        for step in range(steps):
            transits = init.reshape(S, B)[k] if step == 0 else out[k, 0]
            exp = np.concatenate([np.isin(out[k, step], hg.col[hg.row_ptr[t]:hg.row_ptr[t + 1]]) for t in transits])
            assert np.array_equal(rows[k, step, :len(exp)] >= 0, exp) and (rows[k, step, len(exp):] == -1).all()
            found += exp.sum()
    assert found > S * L


@pytest.mark.parametrize("many", [False, True])
def test_fastgcn_tables_of_a_graph(nd, many):
    """A byte of degree per vertex, two where many have 256 neighbours and more, beside the hubs' slots and one bitmap at least."""
    import torch
    V = 1 << 23
    deg = np.zeros(V, np.int64)
    deg[::31 if many else 4096] = 256 if many else 3
    row_ptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    col = (np.arange(row_ptr[-1]) % V).astype(np.int32)
    g = nd.Graph.from_csr(row_ptr, col, np.ones(len(col), np.float32), None)
    torch.cuda.synchronize()
    free, samplers = [torch.cuda.mem_get_info()[0]], []
    for _ in range(3):
        samplers.append(nd.Sampler(g, nd.app_params(8, steps=1, fanout=8, batch=8, seed=3), num_samples=4))
        free.append(torch.cuda.mem_get_info()[0])
    tables = (free[0] - free[1]) - (free[2] - free[3])
    assert tables <= 4 * V + V // 8 + (2 * V + V // 4096 if many else V) + (6 << 20)   # memory comes in pieces of 2 MB


@pytest.mark.parametrize("app,V,B,L", [(8, 20_000, 8, 8), (9, 20_000, 8, 8), (9, 5000, 16, 16), (8, 5000, 40, 33), (8, 5000, 41, 33), (8, 200_000, 32, 32), (9, 200_000, 32, 32),
                                       (9, 200_000, 64, 64), (8, 260_000, 32, 48), (8, 400_000, 64, 64), (9, 400_000, 48, 32)])
def test_layers_by_number_of_samples_and_size(nd, app, V, B, L):
    """Samples share an SM by how many there are, by the layers' size and by the graph's; a sample's layers depend on none of it."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = nd.Graph.rmat(V, 10 * V, seed=1)
    init = np.random.default_rng(V).integers(0, V, (4 * sms + 8) * B).astype(np.int32)

    def job(first, S):
        s = nd.Sampler(g, nd.app_params(app, steps=2, fanout=L, batch=B, seed=3), num_samples=S, first_sample=first, initial=init[first * B:(first + S) * B])
        s.sample()
        aux = s.aux()
        return [x.reshape(S, -1) for x in (s.final_samples(), aux["adj_row"], aux["adj_col"], aux["prob"])]

    one = [np.concatenate(x) for x in zip(*(job(first, sms) for first in range(0, 4 * sms, sms)))]
    for first, S in [(5, sms + 1), (0, 2 * sms), (sms, 2 * sms + sms // 2), (0, 3 * sms), (0, 4 * sms)]:
        got = job(first, S)
        for x, exp in zip(got[:3], one):
            assert np.array_equal(x, exp[first:first + S])
        assert np.allclose(got[3], one[3][first:first + S], rtol=1e-6, atol=0)   # 32-bit results of 64-bit sums in another order


@pytest.mark.parametrize("V,B,L", [(3000, 1, 1), (70_000, 1, 1), (70_000, 4, 16), (70_000, 40, 16), (300_000, 60, 32), (300_000, 150, 32), (300_000, 230, 32)])
@pytest.mark.parametrize("scratch", ["0", "1"])
def test_fastgcn_few_entries(nd, ndo, monkeypatch, V, B, L, scratch):
    """Lists of 0 to 25 entries that begin and end anywhere in eight, with repeated entries, up to and beyond four entries a thread."""
    monkeypatch.setenv("ND_COLLECTIVE_BITMAP_GLOBAL", scratch)
    rng = np.random.default_rng(V + B)
    deg = rng.integers(0, 26, V)
    deg[rng.choice(V, 5, replace=False)] = [V // 100, V // 200, 300, 2100, 255]
    src = np.repeat(np.arange(V), deg).astype(np.int32)
    dst = np.where(rng.random(len(src)) < 0.1, src // 2, rng.integers(0, V, len(src))).astype(np.int32)
    hg = ndo.csr_from_records(src, dst, np.ones(len(src), np.float32), V=V)
    S = 20
    initial = rng.integers(-1, V, S * B).astype(np.int32)
    s = nd.Sampler(nd.Graph.from_csr(hg.row_ptr, hg.col, hg.w, hg.max_w), nd.app_params(8, steps=2, fanout=L, batch=B, seed=3), num_samples=S, initial=initial)
    s.sample()
    exp = ndo.sample(hg, ndo.make_params(8, steps=2, fanout=L, batch=B, seed=3), S, initial=initial)
    aux = s.aux()
    assert np.array_equal(s.final_samples(), exp["out"])   # whole numbers: the sums are exact
    assert np.array_equal(aux["prob"].reshape(-1), exp["prob"].reshape(-1))
    assert np.array_equal(aux["adj_row"], exp["adj_row"]) and np.array_equal(aux["adj_col"], exp["adj_col"])
    assert s.stats()["union_unique"] == exp["counters"]["union_unique"]


@pytest.mark.parametrize("V,B,L", [(2000, 9, 1), (3000, 8, 4), (3000, 9, 4), (3000, 9, 5), (70_000, 65, 5), (70_000, 300, 8), (70_000, 300, 9), (300_000, 700, 3)])
@pytest.mark.parametrize("app", [8, 9])
def test_adjacency_of_short_layers(nd, ndo, app, V, B, L):
    """Few vertices and many lists, repeated ones and ones that are none among them: bit for bit what the lists hold."""
    rng = np.random.default_rng(B + L)
    hg = ndo.rmat_graph(V, 20 * V, seed=3)
    S, steps = 30, 2
    initial = rng.integers(-1, V, S * B).astype(np.int32)
    initial[::7] = initial[3]
    s = nd.Sampler(nd.Graph.from_csr(hg.row_ptr, hg.col, hg.w, hg.max_w), nd.app_params(app, steps=steps, fanout=L, batch=B, seed=3), num_samples=S, initial=initial)
    s.sample()
    out, aux = s.final_samples().reshape(S, steps, L), s.aux()
    rows, cols = aux["adj_row"].reshape(S, steps, -1), aux["adj_col"].reshape(S, steps, -1)
    for k in range(S):
        for step in range(steps):
            transits = initial[k * B:(k + 1) * B] if step == 0 else out[k, step - 1]
            exp = np.zeros((len(transits), L), bool)
            for i, t in enumerate(transits):
                if 0 <= t < V:
                    exp[i] = np.isin(out[k, step], hg.col[hg.row_ptr[t]:hg.row_ptr[t + 1]])
            exp = exp.reshape(-1)
            i, j = np.divmod(np.arange(len(exp)), L)
            assert np.array_equal(rows[k, step, :len(exp)], np.where(exp, i, -1)) and np.array_equal(cols[k, step, :len(exp)], np.where(exp, j, -1))
            assert (rows[k, step, len(exp):] == -1).all()
