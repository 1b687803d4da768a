"""Rows of a caller's pinned array that the GPU writes itself: lines that begin anywhere, shares at whole chunks of rows, rows
that shrink and grow, arrays that turn dense, and a job that starts before the last one's rows are written."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _pinned(n, offset, fill):
    return torch.full((n + offset,), fill, dtype=torch.int32).pin_memory().numpy()[offset:]


@pytest.mark.parametrize("S,steps,offset", [(1 << 14, 7, 0), ((1 << 14) + 1, 100, 1), (20479, 16, 3), (40961, 101, 13), (65536, 5, 5)])
def test_rows_in_pinned_memory(nd, small_graph, S, steps, offset):
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    rng = np.random.default_rng(S)
    out = _pinned(S * steps + 16, offset, g.V)
    out[S * steps:] = -7                                  # behind the array
    row_len = _pinned(S, 0, 0)
    samplers = [nd.Sampler(g, nd.app_params(2, steps=steps, seed=k, stop_prob=p), num_samples=S) for k, p in ((1, 0.3), (2, 0.05), (3, 0.0005))]
    for job in range(7):
        s = samplers[(0, 1, 0, 2, 0, 1, 1)[job]]
        s.set_initial(rng.integers(-1, g.V, S).astype(np.int32))
        s.sample(1)
        exp = s.final_samples()
        s.host_update_begin(out[:S * steps], row_len)
        if job == 4:                                      # the next job of the sampler begins before the rows are written
            s.set_initial(rng.integers(0, g.V, S).astype(np.int32))
            s.sample(1)
        if job >= 5:
            s.host_update_fetch()
        if job == 5:
            s.set_initial(rng.integers(0, g.V, S).astype(np.int32))
            s.sample(1)
        assert s.host_update_finish() >= (exp != g.V).sum()
        assert np.array_equal(out[:S * steps].reshape(S, steps), exp), job
        assert np.array_equal(row_len, (exp != g.V).sum(axis=1)), job
        assert (out[S * steps:S * steps + 16] == -7).all()


@pytest.mark.parametrize("depth", [1, 2])
def test_pipeline_into_pinned_arrays(nd, small_graph, depth):
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    S, rng = 70001, np.random.default_rng(depth)
    pr = nd.app_params(2, steps=40, seed=9, stop_prob=0.15)
    outs = [_pinned(S * 40, k, 0) for k in range(2)]
    streams = torch.cuda.Stream(), torch.cuda.Stream()
    pipe = nd.PipelinedSampler(g, pr, S, chunks=3, depth=depth, stream=streams[0].cuda_stream, copy_stream=streams[1].cuda_stream, sparse_rows=True)
    whole = nd.Sampler(g, pr, num_samples=S)
    seeds = [rng.integers(0, g.V, S).astype(np.int32) for _ in range(6)]
    for k, init in enumerate(seeds):                      # back to back, the arrays in turn and the same one twice
        pipe.run_async(init, outs[(0, 1, 1, 0, 1, 0)[k]])
        if k in (1, 3):
            pipe.wait()
    pipe.wait()
    for out, k in ((outs[0], 5), (outs[1], 4)):
        whole.set_initial(seeds[k])
        whole.sample(1)
        assert np.array_equal(out.reshape(S, 40), whole.final_samples()), k


@pytest.mark.parametrize("depth", [1, 2])
@pytest.mark.parametrize("pinned", [False, True])
def test_an_array_is_forgotten_while_its_rows_are_to_be_written(nd, small_graph, depth, pinned):
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    S, steps, rng = 70_001, 40, np.random.default_rng(depth)
    pr = nd.app_params(2, steps=steps, seed=9, stop_prob=0.15)
    outs = [_pinned(S * steps, 0, 0) if pinned else np.zeros(S * steps, np.int32) for _ in range(2)]
    pipe = nd.PipelinedSampler(g, pr, S, chunks=3, depth=depth, sparse_rows=True)
    whole = nd.Sampler(g, pr, num_samples=S)
    for job in range(6):
        out, init = outs[job % 2], rng.integers(0, g.V, S).astype(np.int32)
        whole.set_initial(init)
        whole.sample(1)
        pipe.run_async(init, out)
        if job in (1, 2, 4):
            pipe.forget(out)                              # the rows are there, and what the caller writes stays
            assert np.array_equal(out.reshape(S, steps), whole.final_samples())
            out[:] = -3
            pipe.wait()
            assert (out == -3).all()
        else:
            pipe.wait()
            assert np.array_equal(out.reshape(S, steps), whole.final_samples())


@pytest.mark.parametrize("step", ["unregistered", "replayed"])
def test_rows_that_the_gpu_may_no_longer_write(nd, small_graph, step):
    """Between the begin and the finish of an update the array stops being pinned, or a captured job runs again."""
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    S, steps, rng = 1 << 14, 40, np.random.default_rng(3)
    s = nd.Sampler(g, nd.app_params(2, steps=steps, seed=5, stop_prob=0.2), num_samples=S)
    rt, page, stream = torch.cuda.cudart(), 4096, torch.cuda.Stream()
    own = np.full(S * steps + 1024, g.V, np.int32)
    out = own[(-own.ctypes.data % page) // 4:][:S * steps]
    row_len = _pinned(S, 0, 0)
    assert int(rt.cudaHostRegister(out.ctypes.data, out.nbytes, 0)) == 0
    s.set_stream(stream.cuda_stream)
    first, second = (rng.integers(0, g.V, S).astype(np.int32) for _ in range(2))
    graph = torch.cuda.CUDAGraph()
    if step == "replayed":
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            s.sample(1, sync=False)
        s.set_initial(first)
        with torch.cuda.stream(stream):
            graph.replay()
    else:
        s.set_initial(first)
        s.sample(1, sync=False)
    expected = s.final_samples().copy()
    s.host_update_begin(out, row_len)
    if step == "replayed":
        s.set_initial(second)
        with torch.cuda.stream(stream):
            graph.replay()
        s.sync()
        assert not np.array_equal(s.final_samples(), expected)
    else:
        stream.synchronize()
        assert int(rt.cudaHostUnregister(out.ctypes.data)) == 0
    s.host_update_finish()
    if step == "replayed":
        assert int(rt.cudaHostUnregister(out.ctypes.data)) == 0
    assert np.array_equal(out.reshape(S, steps), expected)
    assert np.array_equal(row_len, (expected != g.V).sum(axis=1))


def _update(nd, g, S, steps, stop, pinned, app=2):
    s = nd.Sampler(g, nd.app_params(app, steps=steps, seed=5, stop_prob=stop), num_samples=S)
    out, row_len = (_pinned(S * steps, 0, g.V), _pinned(S, 0, 0)) if pinned else (np.full(S * steps, g.V, np.int32), np.zeros(S, np.int32))
    return s, out, row_len


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("stop,mode,then", [(0.2, 1, 1), (0.2, 2, 0), (0.2, 0, 0), (0.0005, 1, 1), (0.0005, 1, 2), (0.0005, 0, 0)])
@pytest.mark.parametrize("between", ["begin and fetch", "fetch and finish"])
def test_the_next_job_at_any_time(nd, small_graph, pinned, stop, mode, then, between):
    """... in a mode that writes the array that the packed rows lie in, and with rows that are mostly full."""
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    S, steps, rng = 20_000, 40, np.random.default_rng(3)
    s, out, row_len = _update(nd, g, S, steps, stop, pinned)
    for _ in range(3):
        s.set_initial(rng.integers(0, g.V, S).astype(np.int32))
        s.sample(mode)
        expected = s.final_samples().copy()
        s.host_update_begin(out, row_len)
        if between == "fetch and finish":
            s.host_update_fetch()
        s.set_initial(rng.integers(0, g.V, S).astype(np.int32))
        s.sample(then, sync=False)
        if between == "begin and fetch":
            s.host_update_fetch()
        s.sync()
        s.host_update_finish()
        assert np.array_equal(out.reshape(S, steps), expected)
        assert np.array_equal(row_len, (expected != g.V).sum(axis=1))


@pytest.mark.parametrize("copy_stream", [False, True])
def test_the_next_job_does_not_wait_on_the_host(nd, small_graph, copy_stream):
    import time
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    S, steps, rng = 1 << 15, 40, np.random.default_rng(3)
    s, out, row_len = _update(nd, g, S, steps, 0.2, True)
    streams = torch.cuda.Stream(), torch.cuda.Stream()
    s.set_stream(streams[0].cuda_stream)
    seeds = [torch.from_numpy(rng.integers(0, g.V, S).astype(np.int32)).pin_memory().numpy() for _ in range(2)]
    for job in range(2):                                  # the second: everything is loaded and allocated
        s.set_initial(seeds[0])
        s.sample(1)
        expected = s.final_samples().copy()
        with torch.cuda.stream(streams[0]):
            torch.cuda._sleep(500_000_000)                # a quarter of a second
        start = time.perf_counter()
        s.host_update_begin(out, row_len, streams[1].cuda_stream if copy_stream else None)
        s.set_initial(seeds[1])
        s.sample(1, sync=False)
        took = time.perf_counter() - start
        assert not streams[0].query() and (job == 0 or took < 0.1), took
        s.host_update_fetch()
        s.host_update_finish()
        s.sync()
        assert np.array_equal(out.reshape(S, steps), expected)


def test_a_job_is_captured_while_an_update_is_open(nd, small_graph):
    g = nd.Graph.from_csr(small_graph.row_ptr, small_graph.col, small_graph.w, small_graph.max_w)
    S, steps, rng = 1 << 15, 40, np.random.default_rng(3)
    s, out, row_len = _update(nd, g, S, steps, 0.2, True)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    s.set_stream(stream.cuda_stream)
    first, second = (rng.integers(0, g.V, S).astype(np.int32) for _ in range(2))
    s.set_initial(first)
    s.sample(1)
    expected = s.final_samples().copy()
    s.host_update_begin(out, row_len)
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        s.sample(1, sync=False)
    s.set_initial(second)
    with torch.cuda.stream(stream):
        graph.replay()
    s.sync()
    replayed = s.final_samples().copy()
    assert not np.array_equal(replayed, expected)
    s.host_update_finish()
    assert np.array_equal(out.reshape(S, steps), expected)
    s.host_update_begin(out, row_len)
    s.host_update_finish()
    assert np.array_equal(out.reshape(S, steps), replayed)
