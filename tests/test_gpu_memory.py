"""Calls that fail for want of device memory: what they leave behind.  The cases that fill the GPU's memory are
processes of their own."""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MB = 1 << 20


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


@pytest.mark.gpu
@pytest.mark.parametrize("app", [0, 4, 9])
def test_a_graph_destroyed_before_its_sampler(nd, small_graph, app):
    """As garbage collection does it with a cycle that holds both."""
    def make():
        g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
        s = nd.Sampler(g, nd.app_params(app, seed=1), num_samples=50)
        s.sample()
        return g, s

    pairs = [make() for _ in range(4)]
    expected = pairs[0][1].final_samples().copy()
    for g, _ in pairs:
        g.free()
    for _, s in pairs:
        s.free()
    assert np.array_equal(make()[1].final_samples(), expected)


class Filled:
    """All but about `left` bytes of the device's memory, allocated and never touched."""

    def __init__(self, left):
        import torch
        torch.cuda.synchronize()
        self.torch, self.held, chunk = torch, [], 1 << 40
        while chunk >= 2 * MB:
            n = min(chunk, torch.cuda.mem_get_info()[0] - left) // (2 * MB) * (2 * MB)
            if n <= 0:
                break
            try:
                self.held.append(torch.empty(n, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                chunk = n // 2

    def free(self):
        self.held.clear()
        self.torch.cuda.empty_cache()


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def samples(nd, graph, app):
    s = nd.Sampler(graph, nd.app_params(app, steps=4 if app < 4 else 2, fanout=8, batch=8, seed=4), num_samples=500)
    s.sample(1)
    return s.final_samples().copy()


# Memory that runs out in the middle of what a graph's first sampler builds: the call fails, nothing it has allocated
# stays behind, and the same call succeeds when there is room again.  What it cannot do without, in MB: DeepWalk 32, node2vec
# 8 + 32 + 256, FastGCN 4 + 30 + 2, LADIES 4 + 30 + 128 + 8; the limits end in the middle of each.
def first_samplers(app):
    from nextdoor_b200 import api as nd
    expected = samples(nd, nd.Graph.rmat(1 << 20, 1 << 24, seed=0), app)   # (and nothing is alive after it: no block is kept)
    graph, failed = nd.Graph.rmat(1 << 20, 1 << 24, seed=0), 0
    for left in (14, 22, 30, 44, 60, 90, 150, 200, 290):
        fill = Filled(left * MB)
        room = []
        for _ in range(4):
            try:
                got = samples(nd, graph, app)
            except nd.NdError as e:
                assert "memory" in str(e), e
                room.append(free_bytes())
                failed += 1
            else:
                fill.free()
                assert np.array_equal(got, expected) and failed >= 4, failed
                return
        assert min(room[1:]) > room[0] - MB, [x / MB for x in room]     # a second failure takes no more (the least array is 4 MB; small ones share pages)
        fill.free()
    assert np.array_equal(samples(nd, graph, app), expected) and failed >= 4


# ids and weights of 64 MB each, row offsets and maxima of 4; the partitioner's arrays of 4, 4, 8 and 8 MB
def graphs_and_partitions(what):
    from nextdoor_b200 import api as nd
    row_ptr, col, w, max_w = nd.Graph.rmat(1 << 20, 1 << 23, seed=0).to_host()
    graph = nd.Graph.from_csr(row_ptr, col, w, max_w) if what == "partition" else None

    def call():
        if graph:
            graph.partition(1 << 20, max_parts=1 << 20)
        else:
            nd.Graph.from_csr(row_ptr, col, w, max_w).free()

    call()
    failed = 0
    for left in (4, 7, 10, 14, 20, 40, 80, 120, 160):
        fill = Filled(left * MB)
        room = []
        for _ in range(4):
            try:
                call()
            except nd.NdError as e:
                assert "memory" in str(e), e
                failed += 1
            room.append(free_bytes())
        assert min(room[1:]) > room[0] - MB, [x / MB for x in room]
        fill.free()
    call()
    assert failed >= 4


# a freed graph's block of 140 MB is kept for the next build, and a sampler needs the room
def kept_blocks():
    from nextdoor_b200 import api as nd
    small = nd.Graph.rmat(1000, 4000, seed=1)
    uniform = nd.app_params(0, steps=100, seed=4)
    s = nd.Sampler(small, uniform, num_samples=1000)
    s.sample()
    expected = s.final_samples().copy()
    nd.Graph.rmat(1 << 20, 1 << 23, seed=0).free()
    fill = Filled(20 * MB)
    assert free_bytes() < 24 * MB
    s = nd.Sampler(small, uniform, num_samples=300_000)          # 120 MB
    s.sample()
    assert np.array_equal(s.final_samples()[:1000], expected)
    fill.free()


# the adjacency of 102 M entries crosses as 13 MB of bits, which do not fit: it is copied as it is
def adjacency():
    from nextdoor_b200 import api as nd
    graph = nd.Graph.rmat(20_000, 80_000, seed=1)
    s, t = (nd.Sampler(graph, nd.app_params(6, steps=5, seed=2), num_samples=5000) for _ in range(2))
    s.sample()
    t.sample()
    expected = t.aux()
    fill = Filled(6 * MB)
    got = s.aux()
    fill.free()
    assert (got["adj_row"] >= 0).any()
    assert np.array_equal(got["adj_row"], expected["adj_row"]) and np.array_equal(got["adj_col"], expected["adj_col"])


# pinned memory for the rows of a job (16 MB and more) that the process may not have: the update fails, the next one works
def pinned_rows():
    import resource
    from nextdoor_b200 import api as nd
    graph = nd.Graph.rmat(1 << 18, 1 << 21, seed=1)
    S, steps = 1 << 20, 50
    s = nd.Sampler(graph, nd.app_params(2, steps=steps, seed=2, stop_prob=0.1), num_samples=S)
    out, row_len = np.full(S * steps, graph.V, np.int32), np.zeros(S, np.int32)
    seeds = (np.arange(S) % graph.V).astype(np.int32)

    def update(initial):
        s.set_initial(initial)
        s.sample(1)
        s.host_update_begin(out, row_len)
        s.host_update_fetch()
        s.host_update_finish()

    update(np.full(S, -1, np.int32))             # no rows: everything but their memory is there
    old = resource.getrlimit(resource.RLIMIT_AS)
    pages = int(open("/proc/self/statm").read().split()[0])
    resource.setrlimit(resource.RLIMIT_AS, (pages * resource.getpagesize() + 8 * MB, old[1]))
    try:
        with pytest.raises(nd.NdError, match="memory"):
            update(seeds)
    finally:
        resource.setrlimit(resource.RLIMIT_AS, old)
    update(seeds)
    assert np.array_equal(out.reshape(S, steps), s.final_samples())


# a load needs no more memory where its ids are sorted while the weights are on the wire, from 2^21 records on
def loads():
    from nextdoor_b200 import api as nd
    rng, n, V = np.random.default_rng(1), 1 << 21, 1 << 18
    src, dst, w = rng.integers(0, V, n).astype(np.int32), rng.integers(0, V, n).astype(np.int32), rng.random(n).astype(np.float32)
    src[0] = V - 1
    need = []
    for k in (n - 1, n):
        lo, hi = 0, 256
        while hi - lo > 1:
            mid = (lo + hi) // 2
            fill = Filled(mid * MB)
            try:
                nd.Graph.from_edge_records(src[:k], dst[:k], w[:k]).free()
                hi = mid
            except nd.NdError as e:
                assert "memory" in str(e), e
                lo = mid
            fill.free()
        need.append(hi)
    assert 60 < need[0] < 256 and need[1] <= need[0] + 4, need    # MB: three words a record twice, the graph; memory comes in pages of 2


# What a first sampler builds only to be faster (the last of it: entries of 64 MB, ids of 48, ids with weights of 128 and 64, tables of the hubs) and finds no
# room for, it does without
def without_the_last(app, vertices, edges, spare):
    from nextdoor_b200 import api as nd
    graph = nd.Graph.rmat(vertices, edges, seed=0)
    rows, expected = graph.to_host(), samples(nd, graph, app)
    graph.free()
    graph = nd.Graph.from_csr(*rows)
    before = free_bytes()
    assert np.array_equal(samples(nd, graph, app), expected)
    built = before - free_bytes()
    graph.free()
    assert built > 3 * spare * MB, built / MB
    graph = nd.Graph.from_csr(*rows)
    fill = Filled(built - spare * MB)
    assert free_bytes() < built
    got = samples(nd, graph, app)
    fill.free()
    assert np.array_equal(got, expected)
    assert np.array_equal(samples(nd, graph, app), expected)


@pytest.mark.gpu
@pytest.mark.parametrize("app,vertices,edges,spare", [(0, 1 << 18, 1 << 21, 8), (0, 1 << 20, 1 << 24, 8), (1, 1 << 18, 1 << 21, 8), (9, 1 << 20, 1 << 24, 8),
                                                         (1, 1 << 20, 1 << 24, 8), (2, 1 << 22, 1 << 23, 8)])
def test_a_sampler_without_room_for_what_is_optional(app, vertices, edges, spare):
    case = f"without_the_last({app}, {vertices}, {edges}, {spare})"
    r = subprocess.run([sys.executable, os.path.abspath(__file__), case], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


@pytest.mark.gpu
@pytest.mark.parametrize("case", [f"first_samplers({app})" for app in (1, 3, 8, 9)]
                         + [f"graphs_and_partitions('{what}')" for what in ("csr", "partition")] + ["kept_blocks()", "adjacency()", "pinned_rows()", "loads()"])
def test_nothing_stays_behind(case):
    r = subprocess.run([sys.executable, os.path.abspath(__file__), case], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


if __name__ == "__main__":
    sys.path.insert(0, ROOT)
    eval(sys.argv[1])
