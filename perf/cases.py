"""Performance cases: the calls a program built on this package spends its time in.

Six kinds of work, each through the public entry points:

``propagate``  compressed propagation of a feature matrix (``Compressgnn_SPMM``), inference or
               forward + backward: the operator every model layer starts with.
``refresh``    the bucket assignment of ``Compressgnn_Cluster`` for features that moved.
``transform``  ``Compressgnn_Cluster`` -> ``Linear`` -> ``Compressgnn_Reconstruct``, forward + backward, the
               assignment reused for five epochs: a layer's transformation half on its own.
``model``      the ``GCN`` stack: a training step up to the gradients (the optimiser is torch's), or inference.
``sample``     mini-batches of seed nodes, neighbours sampled hop by hop on the compressed graph.
``compress``   grammar compression of a graph, host arrays in and host arrays out (graph preparation).

Graphs come from the package's copying-model web generator with the parameters of the benchmark.  A graph
is a data set: its host arrays depend on the size only and are made once per process; features,
gradients, labels, weights, planes and seed nodes come from the seed, and so does the order of the rows
that ``compress`` is given (the rules found do not depend on it, so every order has outputs of one size).
"""
import functools
import math

import numpy as np
import torch

from compressgnn_b200 import offline
from compressgnn_b200.layer import Compressgnn_Cluster, Compressgnn_Reconstruct, Compressgnn_SPMM
from compressgnn_b200.loader import CompressGraph, compress, compress_graph_csr
from compressgnn_b200.model import GCN

WEB_NODES = 325557      # nodes of the benchmark's web graph (3.1 M edges)
LARGE_NODES = 2450000   # nodes of the benchmark's cluster workload
CENTROIDS = 4096        # directions the clustered features scatter around
REFRESH = 5             # epochs an assignment is kept


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # citation-graph sized inputs: launches and host time are all there is
        dict(name="propagate-small", kind="propagate", nodes=2708, width=16, dtype="f32", train=True),
        # the benchmark's headline workload
        dict(name="propagate-web", kind="propagate", nodes=WEB_NODES, width=256, dtype="f32", train=True),
        # the same graph with one quarter of the columns (hidden layers, column shards), inference
        dict(name="propagate-web-narrow", kind="propagate", nodes=WEB_NODES, width=64, dtype="f32", train=False),
        # raw features of a width that is no multiple of four
        dict(name="propagate-ragged", kind="propagate", nodes=40000, width=602, dtype="f32", train=True),
        # double precision, as for gradient checks and sensitive solvers
        dict(name="propagate-double", kind="propagate", nodes=40000, width=128, dtype="f64", train=True),
        # the refresh epoch of the benchmark's cluster workload
        dict(name="refresh-large", kind="refresh", nodes=LARGE_NODES, width=128, bits=16, dtype="f32"),
        # the benchmark's cluster workload
        dict(name="transform-large", kind="transform", nodes=LARGE_NODES, width=128, out=256, bits=16, dtype="f32",
             relu=True),
        # full-batch training on a citation-sized graph: two layers, 64 hidden, 7 classes
        dict(name="train-small", kind="model", nodes=2708, width=128, hidden=64, classes=7, layers=2,
             transform=True, train=True),
        # full-batch training on the web graph: the benchmark's end-to-end workload
        dict(name="train-web", kind="model", nodes=WEB_NODES, width=256, hidden=128, classes=47, layers=2,
             transform=True, train=True),
        # scoring every node of the web graph from wide raw features
        dict(name="infer-web-wide", kind="model", nodes=WEB_NODES, width=1024, hidden=128, classes=47, layers=2,
             transform=True, train=False),
        # mini-batches as GraphSAGE-style loaders draw them
        dict(name="sample-web", kind="sample", nodes=WEB_NODES, batch=1024, hop1=25, hop2=10, hop3=0),
        # compressing the web graph when it is loaded
        dict(name="compress-web", kind="compress", nodes=WEB_NODES, frequency=4),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("propagate", "propagate", "refresh", "transform", "model", "model", "sample", "compress"))
    if kind == "propagate":
        nodes = _log_int(rng, 1000, WEB_NODES)
        double = rng.random() < 0.2
        most = WEB_NODES * 256 // (nodes * (2 if double else 1))
        return dict(kind=kind, nodes=nodes, width=_log_int(rng, 1, min(1024, most)),
                    dtype="f64" if double else "f32", train=rng.random() < 0.6)
    if kind in ("refresh", "transform"):
        nodes = _log_int(rng, 2000, LARGE_NODES)
        double = rng.random() < 0.15
        most = LARGE_NODES * 128 // (nodes * (2 if double else 1))
        case = dict(kind=kind, nodes=nodes, width=_log_int(rng, 8, max(8, min(1024, most))), bits=rng.randint(4, 20),
                    dtype="f64" if double else "f32")
        if kind == "transform":
            case.update(out=_log_int(rng, 8, max(8, min(512, 2 * most))), relu=rng.random() < 0.7)
        return case
    if kind == "model":
        return dict(kind=kind, nodes=_log_int(rng, 1000, WEB_NODES), width=_log_int(rng, 16, 512),
                    hidden=rng.choice((16, 64, 128, 256)), classes=rng.randint(2, 64), layers=rng.choice((2, 2, 3)),
                    transform=rng.random() < 0.75, train=rng.random() < 0.7)
    if kind == "sample":
        return dict(kind=kind, nodes=_log_int(rng, 5000, WEB_NODES), batch=_log_int(rng, 64, 4096),
                    hop1=rng.randint(5, 25), hop2=rng.randint(5, 15), hop3=rng.choice((0, 0, 5)))
    return dict(kind=kind, nodes=_log_int(rng, 2000, WEB_NODES), frequency=rng.randint(4, 16))


# ---------------------------------------------------------------------------------------------
# graphs
# ---------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def _web_graph(nodes):
    vlist, elist = offline.generate_copy_graph(nodes, alpha=2.1, x_min=5.3, max_degree=10000, copy_prob=0.7,
                                               window=64, candidates=8, seed=2)
    return offline.add_self_loop_csr(vlist, elist)


@functools.lru_cache(maxsize=8)
def _compressed(nodes):
    """The normalised, compressed, transposed web graph as ``CompressGraph`` takes it."""
    vlist, elist = _web_graph(nodes)
    norm = offline.get_norm_degree(elist, nodes)
    cv, ce, vertices, rules = compress(vlist, elist, 4, 3, 1000000, min_pair_frequency=4)
    cv, ce = cv.astype(np.int64), ce.astype(np.int64)
    weight = offline.gcn_norm_csr_compress(cv, ce, norm, vertices, rules)
    return offline.transpose_csr(cv, ce, weight, vertices + rules), int(rules), int(elist.size)


def _graph(nodes):
    (vlist, elist, weight), _, _ = _compressed(nodes)
    return CompressGraph(vlist, elist, weight, nodes).to("cuda")


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def _dtype(case):
    return torch.float64 if case.get("dtype") == "f64" else torch.float32


def _clustered(nodes, width, dtype, gen):
    centroids = torch.randn(CENTROIDS, width, device="cuda", dtype=dtype, generator=gen)
    which = torch.randint(0, CENTROIDS, (nodes,), device="cuda", generator=gen)
    return centroids[which].add_(torch.randn(nodes, width, device="cuda", dtype=dtype, generator=gen), alpha=0.1)


def prepare(case, seed):
    torch.manual_seed(seed)  # weights, planes and the dropout of a training step
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, nodes, dtype = case["kind"], case["nodes"], _dtype(case)
    state = dict(case=case)
    if kind == "propagate":
        state.update(graph=_graph(nodes), spmm=Compressgnn_SPMM(),
                     x=torch.randn(nodes, case["width"], device="cuda", dtype=dtype, generator=gen))
        if case["train"]:
            state["x"].requires_grad_()
            state["grad"] = torch.randn(nodes, case["width"], device="cuda", dtype=dtype, generator=gen)
    elif kind == "refresh":
        state.update(x=_clustered(nodes, case["width"], dtype, gen), epoch=0,
                     cluster=Compressgnn_Cluster(case["width"], case["bits"], device="cuda", dtype=dtype))
    elif kind == "transform":
        state.update(x=_clustered(nodes, case["width"], dtype, gen).requires_grad_(), epoch=0,
                     cluster=Compressgnn_Cluster(case["width"], case["bits"], device="cuda", dtype=dtype,
                                                 refresh_interval=REFRESH),
                     lin=torch.nn.Linear(case["width"], case["out"]).to(device="cuda", dtype=dtype),
                     reconstruct=Compressgnn_Reconstruct(),
                     grad=torch.randn(nodes, case["out"], device="cuda", dtype=dtype, generator=gen))
    elif kind == "model":
        model = GCN(case["width"], case["classes"], hidden_features=case["hidden"], param_H=16, dropout=0.3,
                    use_transformation=case["transform"], refresh_interval=REFRESH, num_layers=case["layers"]).cuda()
        state.update(graph=_graph(nodes), model=model.train(case["train"]), epoch=0,
                     x=torch.randn(nodes, case["width"], device="cuda", generator=gen),
                     labels=torch.randint(0, case["classes"], (nodes, 1), device="cuda", generator=gen))
    elif kind == "sample":
        batches = [torch.randperm(nodes, device="cuda", generator=gen)[:case["batch"]].clone() for _ in range(8)]
        hops = [h for h in (case["hop1"], case["hop2"], case["hop3"]) if h]
        edges = sum(case["batch"] * math.prod(hops[:i + 1]) for i in range(len(hops)))
        # a mini-batch is handed on in buffers of a fixed size, which the layers behind it are compiled for
        buffers = [torch.full((most,), -1, device="cuda") for most in (case["batch"] + edges, edges, edges)]
        state.update(sampler=_graph(nodes).neighbor_sampler(), batches=batches, seed=seed, at=0, hops=hops,
                     buffers=buffers)
    else:
        vlist, elist = _web_graph(nodes)
        first = int(np.random.default_rng(seed).integers(1, nodes))  # the row that comes first
        lengths = np.roll(np.diff(vlist), -first)
        state["vlist"] = np.concatenate([np.zeros(1, np.int64), np.cumsum(lengths)])
        state["elist"] = np.roll(elist, -int(vlist[first]))
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "propagate":
        if not case["train"]:
            with torch.no_grad():
                return state["spmm"](state["graph"], state["x"])
        x = state["x"]
        x.grad = None
        out = state["spmm"](state["graph"], x)
        out.backward(state["grad"])
        return out.detach(), x.grad
    if kind == "refresh":
        cluster = state["cluster"]
        cluster.set_epoch(state["epoch"])
        state["epoch"] += 1
        found = cluster.assignment(state["x"])
        return found.index, found.active
    if kind == "transform":
        x, lin = state["x"], state["lin"]
        x.grad = lin.weight.grad = lin.bias.grad = None
        state["cluster"].set_epoch(state["epoch"])
        state["epoch"] += 1
        reps, index = state["cluster"](x)
        out = state["reconstruct"](torch.nn.functional.linear(reps, lin.weight, None), index, bias=lin.bias,
                                   activation="relu" if case["relu"] else None)
        out.backward(state["grad"])
        return out.detach(), x.grad, lin.weight.grad, lin.bias.grad
    if kind == "model":
        model = state["model"]
        model.set_epoch(state["epoch"])
        state["epoch"] += 1
        if not case["train"]:
            with torch.no_grad():
                return model.inference(state["x"], state["graph"])
        model.zero_grad(set_to_none=True)
        scores = model(state["x"], state["graph"])
        loss = -scores.gather(1, state["labels"]).mean()
        loss.backward()
        return [scores.detach(), loss.detach()] + [p.grad for p in model.parameters()]
    if kind == "sample":
        batch = state["batches"][state["at"] % len(state["batches"])]
        state["at"] += 1
        found = state["sampler"](batch, state["hops"], seed=state["seed"])
        for buffer, part in zip(state["buffers"], found):
            buffer[:part.numel()].copy_(part)
        return state["buffers"], found[0].numel(), found[1].numel()
    return compress_graph_csr(state["vlist"], state["elist"], case["frequency"], backend="cuda")


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _propagation_work(nodes, width, size):
    """One direction: the matrix read and the result written, and per entry of the compressed graph a column,
    a value and one multiply-add per feature."""
    (vlist, elist, _), _, _ = _compressed(nodes)
    return 2 * size * nodes * width + 8 * elist.size + 4 * vlist.size, 2 * elist.size * width


def _transform_work(nodes, width, out, size, backward, input_grad, groups):
    """Features averaged per bucket, a Linear on the averages, the result spread; backward the same in reverse."""
    nbytes = size * nodes * (width + out) + 8 * nodes + size * width * out
    flops = nodes * (width + out) + 2 * groups * width * out
    if backward:
        nbytes += size * nodes * (out + (width if input_grad else 0)) + 2 * size * width * out
        flops += nodes * out + 2 * groups * width * out * (2 if input_grad else 1)
    return nbytes, flops


def work(case):
    kind, nodes = case["kind"], case["nodes"]
    size = 8 if case.get("dtype") == "f64" else 4
    nbytes = flops = 0
    if kind == "propagate":
        b, f = _propagation_work(nodes, case["width"], size)
        times = 2 if case["train"] else 1
        nbytes, flops = times * b, times * f
    elif kind == "refresh":
        nbytes = size * nodes * case["width"] + 8 * nodes + size * case["width"] * case["bits"]
        flops = 2 * nodes * case["width"] * case["bits"]
    elif kind == "transform":
        groups = min(nodes, CENTROIDS, 2 ** case["bits"])
        nbytes, flops = _transform_work(nodes, case["width"], case["out"], size, True, True, groups)
    elif kind == "model":
        dims = [case["width"]] + [case["hidden"]] * (case["layers"] - 1) + [case["classes"]]
        groups = min(nodes, 2 ** 16) if case["transform"] else nodes
        for i, (a, b) in enumerate(zip(dims, dims[1:])):
            both = case["train"] and i > 0  # the input features take no gradient
            pb, pf = _propagation_work(nodes, a, size)
            tb, tf = _transform_work(nodes, a, b, size, case["train"], both, groups)
            nbytes += pb * (2 if both else 1) + tb
            flops += pf * (2 if both else 1) + tf
    elif kind == "sample":
        frontier, edges = case["batch"], 0
        for hop in (case["hop1"], case["hop2"], case["hop3"]):
            frontier = min(frontier, nodes) * min(hop, 9)  # the mean degree bounds what a node contributes
            edges += frontier
        nbytes, flops = 8 * (case["batch"] + 4 * edges), edges  # the graph's column, and three values out
    else:
        edges = 10 * nodes
        nbytes, flops = 8 * (nodes + edges) + 4 * (nodes + edges), edges
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind in ("refresh", "sample", "compress"):
        return "exact"
    if case.get("dtype") == "f64":
        return {"rel": 1e-12}
    if kind == "model":
        # A sum rounded another way moves the features of a hidden layer by about 1e-6, which puts up to
        # 1e-6 * 16 planes of the nodes on the other side of a hyperplane: into another bucket, with other
        # scores, and the other nodes of both buckets move with their means.  Twice the root of that share is
        # what two correct implementations differ by, and single values of those nodes differ entirely.
        return {"rel": 1e-2, "max": 0.99} if case["transform"] else {"rel": 1e-4, "max": 0.5}
    if kind == "transform" and case["relu"]:
        # a pre-activation within rounding (1e-7) of zero has its gradient masked or not: again the root of
        # the share, and the whole of a single value
        return {"rel": 5e-4, "max": 0.99}
    return {"rel": 1e-5}
