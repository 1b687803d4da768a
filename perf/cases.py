"""The calls whose time matters to a user of this framework, with inputs of the shapes it is used on.

A case is one job through the public entry points (`nextdoor_b200.api`, `nextdoor_b200.dist`):

* `walk`          uniform / DeepWalk / PPR / node2vec walks that stay on the GPU for the next consumer (embedding
                  training): `Sampler.sample()` in its default mode and the zero-copy device tensor;
* `walk_module`   the calls behind the reference's Python module: `sample()` in the module's sample-parallel mode on
                  the default stream, then the final samples as a host array;
* `walk_host`     host seeds in, dense host array out, through `PipelinedSampler`;
* `khop`          GraphSAGE neighbourhoods of a whole set of seeds at once;
* `khop_batch`    a training loader's mini-batch: new seeds from the host for every call, on the loader's own stream;
* `layer`         FastGCN / LADIES layers, samples on the device; with `"aux"` also the adjacency entries and the
                  probabilities, which the API hands out as host arrays;
* `layer_module`  the reference's shipped FastGCN / LADIES applications as its Python module runs them;
* `load`          12-byte edge records in host memory to a graph in GPU memory.

Graphs are R-MAT (.57, .19, .19, .05), symmetrised, weights uniform [1, 5): what the framework's benchmark and tests
use in place of the public graphs.  A sampler's random draws are keyed by its seed, so all integer results are exact.
"""
import ctypes

import numpy as np
import torch

from nextdoor_b200 import api as nd
from nextdoor_b200 import dist as nd_dist

APPS = {"uniform": nd.APP_UNIFORM_WALK, "deepwalk": nd.APP_DEEPWALK, "ppr": nd.APP_PPR, "node2vec": nd.APP_NODE2VEC,
        "khop": nd.APP_KHOP, "khop_distinct": nd.APP_KHOP_DISTINCT, "fastgcn_ref": nd.APP_FASTGCN_REF,
        "ladies_ref": nd.APP_LADIES_REF, "fastgcn": nd.APP_FASTGCN_IS, "ladies": nd.APP_LADIES_IS}


def listed():
    return [
        # a mini-batch of a GraphSAGE loader: 1024 seeds, 25 then 10 neighbours; launches and latency count
        {"name": "khop_batch_1024", "kind": "khop_batch", "app": "khop", "V": 1 << 21, "M": 1 << 25, "S": 1024, "fanout": "25,10"},
        # the same neighbourhoods without replacement for 256 batches in one job, each hop deduplicated
        {"name": "khop_distinct_256k", "kind": "khop", "app": "khop_distinct", "V": 1 << 21, "M": 1 << 25, "S": 1 << 18, "fanout": "25,10"},
        # DeepWalk's uniform walks on a graph of PPI's size: little work per step, a long chain of steps
        {"name": "uniform_57k", "kind": "walk", "app": "uniform", "V": 56944, "M": 400_000, "S": 56944, "steps": 100, "stream": True},
        # ... and as the Python module hands them to a host program
        {"name": "uniform_57k_module", "kind": "walk_module", "app": "uniform", "V": 56944, "M": 400_000, "S": 56944, "steps": 100},
        # weighted and second-order walks, one per vertex of a million-vertex graph: the ordinary training corpus
        {"name": "deepwalk_1m", "kind": "walk", "app": "deepwalk", "V": 1 << 20, "M": 1 << 24, "S": 1 << 20, "steps": 100, "stream": True},
        {"name": "node2vec_1m", "kind": "walk", "app": "node2vec", "V": 1 << 20, "M": 1 << 24, "S": 1 << 20, "steps": 100, "p": 2.0, "q": 0.5, "stream": True},
        # personalised PageRank walks (stop probability 0.15) of a 2^24-vertex, 537 M-entry graph: the largest job
        {"name": "ppr_16m", "kind": "walk", "app": "ppr", "V": 1 << 24, "M": 1 << 28, "S": 1 << 24, "steps": 100, "stop": 0.15, "stream": True},
        # ... and end to end for a host program, seeds in and dense rows out
        {"name": "ppr_2m_host", "kind": "walk_host", "app": "ppr", "V": 1 << 21, "M": 1 << 25, "S": 1 << 21, "steps": 100, "stop": 0.15},
        # importance-sampled layers for 1024 batches of 64 seeds
        {"name": "fastgcn_1k", "kind": "layer", "app": "fastgcn", "V": 1 << 20, "M": 1 << 24, "S": 1024, "B": 64, "L": 64, "steps": 2, "aux": False},
        {"name": "ladies_1k_aux", "kind": "layer", "app": "ladies", "V": 1 << 20, "M": 1 << 24, "S": 1024, "B": 64, "L": 64, "steps": 2, "aux": True},
        # the reference's FastGCN application with its own constants (10,000 samples, 5 layers of 64)
        {"name": "fastgcn_ref_10k", "kind": "layer_module", "app": "fastgcn_ref", "V": 56944, "M": 400_000, "S": 10_000, "B": 64, "L": 64, "steps": 5},
        # loading a graph from an edge list that lies in host memory
        {"name": "load_8m", "kind": "load", "V": 1 << 19, "M": 1 << 22},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["walk", "walk", "walk", "walk_module", "walk_host", "khop", "khop_batch", "layer", "layer_module", "load"])
    if kind == "load":
        V = _log(rng, 1 << 15, 1 << 20)
        return {"kind": kind, "V": V, "M": V * rng.randint(4, 12)}
    if kind == "khop_batch":
        V = _log(rng, 1 << 16, 1 << 22)
        return {"kind": kind, "app": rng.choice(["khop", "khop_distinct"]), "V": V, "M": V * rng.randint(8, 16), "S": _log(rng, 64, 8192),
                "fanout": rng.choice(["25,10", "10,10", "15,10", "5,5", "10,5,5"])}
    if kind == "khop":
        V = _log(rng, 1 << 16, 1 << 22)
        return {"kind": kind, "app": rng.choice(["khop", "khop_distinct"]), "V": V, "M": V * rng.randint(8, 16), "S": _log(rng, 1 << 14, 1 << 18),
                "fanout": rng.choice(["25,10", "10,10", "15,10", "20,3", "10,5,5"])}
    if kind == "layer":
        V = _log(rng, 1 << 16, 1 << 20)
        return {"kind": kind, "app": rng.choice(["fastgcn", "ladies"]), "V": V, "M": V * rng.randint(8, 16), "S": _log(rng, 64, 1024),
                "B": rng.choice([32, 64, 100]), "L": rng.choice([32, 64, 100]), "steps": rng.randint(2, 3), "aux": rng.random() < 0.5}
    if kind == "layer_module":
        V = _log(rng, 1 << 15, 1 << 20)
        return {"kind": kind, "app": rng.choice(["fastgcn_ref", "ladies_ref"]), "V": V, "M": V * rng.randint(4, 12), "S": _log(rng, 1000, 10_000),
                "B": rng.choice([32, 64]), "L": 64, "steps": rng.randint(2, 5)}
    if kind == "walk_module":
        V = _log(rng, 1 << 14, 1 << 18)
        return {"kind": kind, "app": rng.choice(["uniform", "deepwalk", "node2vec"]), "V": V, "M": V * rng.randint(4, 16), "S": V,
                "steps": rng.randint(10, 100), "p": 2.0, "q": 0.5}
    if kind == "walk_host":
        V = _log(rng, 1 << 16, 1 << 21)
        return {"kind": kind, "app": "ppr", "V": V, "M": V * rng.randint(8, 16), "S": V, "steps": rng.randint(40, 100), "stop": rng.choice([0.1, 0.15, 0.2])}
    V = _log(rng, 1 << 15, 1 << 22)
    c = {"kind": kind, "app": rng.choice(["uniform", "deepwalk", "ppr", "node2vec"]), "V": V, "M": V * rng.randint(7, 16),
         "S": V, "steps": rng.randint(40, 100), "stream": rng.random() < 0.7}
    if c["app"] == "ppr":
        c["stop"] = rng.choice([0.1, 0.15, 0.2])
    if c["app"] == "node2vec":
        c["p"], c["q"] = rng.choice([(2.0, 0.5), (1.0, 1.0), (0.5, 2.0), (4.0, 0.25)])
    return c


def _params(case, seed):
    app = APPS[case["app"]]
    if "fanout" in case:
        return nd.app_params(app, fanout=[int(f) for f in case["fanout"].split(",")], seed=seed)
    if "L" in case:
        return nd.app_params(app, steps=case["steps"], fanout=case["L"], batch=case["B"], seed=seed)
    return nd.app_params(app, steps=case["steps"], seed=seed, stop_prob=case.get("stop", 0.01), p=case.get("p", 2.0), q=case.get("q", 0.5))


class _Device:
    """Device memory of the library as an array other packages can read in place, and which keeps its owner alive."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3}


def _csr_tensors(graph):
    ptr = [ctypes.c_void_p() for _ in range(4)]
    nd.check(nd.lib.nd_graph_device_ptrs(graph._h, *[ctypes.byref(p) for p in ptr]))
    sizes = ((graph.V + 1, "<i4"), (graph.E, "<i4"), (graph.E, "<f4"), (graph.V, "<f4"))
    return [torch.as_tensor(_Device(graph, p.value, n, t), device="cuda") for p, (n, t) in zip(ptr, sizes)]


def _samples(sampler):
    """The final samples where they lie; the tensor is a view of the sampler's buffer, which has to outlive it."""
    out = nd_dist.device_samples(sampler)
    out.sampler = sampler
    return out


def _edge_records(case, seed):
    """The records of an R-MAT graph in the order of a file that nobody sorted."""
    graph = nd.Graph.rmat(case["V"], case["M"], seed=seed)
    row_ptr, col, w, _ = _csr_tensors(graph)
    src = torch.repeat_interleave(torch.arange(graph.V, dtype=torch.int32, device="cuda"), (row_ptr[1:] - row_ptr[:-1]).long())
    gen = torch.Generator(device="cuda").manual_seed(seed)
    order = torch.randperm(graph.E, device="cuda", generator=gen)
    src, col, w = [x[order].cpu().numpy() for x in (src, col, w)]
    src[0] = case["V"] - 1                               # the loader counts vertices by the largest id: the last one has an edge
    return [src, col, w]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "load":
        return {"kind": kind, "records": _edge_records(case, seed)}
    graph = nd.Graph.rmat(case["V"], case["M"], seed=seed)
    params, S = _params(case, seed), case["S"]
    rng = np.random.default_rng(seed)
    st = {"kind": kind}
    if kind == "walk_host":
        streams = torch.cuda.Stream(), torch.cuda.Stream()
        st["streams"] = streams
        st["seeds"] = torch.arange(S, dtype=torch.int32).pin_memory().numpy()
        st["out"] = torch.empty(S * case["steps"], dtype=torch.int32, pin_memory=True).numpy()
        st["pipe"] = nd.PipelinedSampler(graph, params, S, initial=st["seeds"], stream=streams[0].cuda_stream,
                                         copy_stream=streams[1].cuda_stream, sparse_rows=True)
        return st
    if kind in ("walk", "walk_module", "layer_module"):
        initial = None                                   # one walk per vertex; batches of consecutive ids
    else:
        initial = rng.integers(0, graph.V, S * nd.initial_sample_size(params)).astype(np.int32)
    st["sampler"] = nd.Sampler(graph, params, num_samples=S, initial=initial)
    if kind == "khop_batch" or case.get("stream"):
        st["stream"] = torch.cuda.Stream()
        st["sampler"].set_stream(st["stream"].cuda_stream)
    if kind == "khop_batch":                             # the next batch, in pinned memory as a loader keeps it
        st["seeds"] = torch.from_numpy(rng.integers(0, graph.V, S).astype(np.int32)).pin_memory().numpy()
    if kind == "layer":
        st["aux"] = case["aux"]
    return st


def run(state):
    kind = state["kind"]
    if kind == "load":
        src, dst, w = state["records"]
        state["graph"] = nd.Graph.from_edge_records(src, dst, w)
        return _csr_tensors(state["graph"])
    if kind == "walk_host":
        state["pipe"].run(state["seeds"], state["out"])
        return state["out"]
    sampler = state["sampler"]
    if kind == "khop_batch":                             # enqueued on the loader's stream; the training step that follows waits for it there
        sampler.set_initial(state["seeds"])
        sampler.sample(sync=False)
        return _samples(sampler)
    if kind == "walk_module":
        sampler.sample(nd.MODE_SAMPLE_PARALLEL)
        return sampler.final_samples()
    sampler.sample()
    if kind == "layer_module":
        return sampler.final_samples()
    out = _samples(sampler)
    if kind == "layer" and state["aux"]:
        aux = sampler.aux()
        return [out, aux["adj_row"], aux["adj_col"], aux["prob"]]
    return out


def _edges(case):
    """About how many vertices one pass samples (an upper bound where walks or neighbour lists end early)."""
    if "fanout" in case:
        n, total = 1, 0
        for f in case["fanout"].split(","):
            n *= int(f)
            total += n
        return case["S"] * total
    if "L" in case:
        return case["S"] * case["steps"] * case["L"]
    steps = case["steps"]
    return case["S"] * (min(steps, (1 - case["stop"]) / case["stop"]) if "stop" in case else steps)


def work(case):
    V, E = case["V"], 2 * case["M"]
    if case["kind"] == "load":                           # records in, row offsets, ids, weights and per-vertex maxima out
        return {"bytes": 12 * E + 8 * E + 8 * V, "flops": 0}
    n = _edges(case)
    weighted = case["app"] in ("deepwalk", "ppr", "ladies")
    graph = 4 * V + min(E, n) * (8 if weighted else 4)   # row offsets; the entries it can touch, each once
    if "L" not in case:                                  # seeds in, one vertex per sampled edge out
        return {"bytes": graph + 4 * case["S"] + 4 * n, "flops": 0}
    S, B, L, steps = case["S"], case["B"], case["L"], case["steps"]
    if not case["app"].endswith("_ref"):                 # every neighbour list of a batch and of its first layers is read
        graph = 4 * V + E * (8 if weighted else 4)
    adjacency = 8 * S * steps * max(B, L) * L
    return {"bytes": graph + 4 * S * B + 8 * n + adjacency, "flops": 0}


def tolerance(case):
    """Vertices, rows and edges follow from keyed 32-bit draws: exact.  Importance sampling sums weights in 64 bits and
    reports 32-bit probabilities; a draw on the very edge of an interval may fall to its neighbour."""
    if case.get("app") in ("fastgcn", "ladies"):
        return {"rel": 1e-5, "differ": 1e-3}
    return "exact"
