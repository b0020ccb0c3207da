"""Performance cases of the sampling framework: what a training or inference program asks of it, call by call.

Every case draws a synthetic power-law graph in int64 CSC from its seed (the real datasets are not available offline),
prepares what such a program holds before the call — the loaded graph, edge weights, features, seed nodes — and runs one
pass through the public entry points (`graph_sampling_b200.gs` and `graph_sampling_b200.ops`).
"""
import math
import random

import numpy as np
import torch

import graph_sampling_b200.gs as gs
from graph_sampling_b200 import ops

# Node of popularity rank r has weight ~ (r + shift)^-SKEW: in-degree and the chance to be somebody's neighbour follow it,
# so the frontier of a hop is made of hubs, as in the graphs these samplers run on.
SKEW = 0.75
CHUNK = 1 << 26  # edges generated at a time
SHAPE_SEED = 20_240
DRAW_SEED = 7


# ---- cases -----------------------------------------------------------------------------------------------------------------
def listed():
    small = {"nodes": 100_000, "edges": 2_000_000}
    products = {"nodes": 2_450_000, "edges": 123_700_000}
    layered = {"nodes": 1_000_000, "edges": 50_000_000}
    papers = {"nodes": 111_000_000, "edges": 1_600_000_000}
    return [
        # a training loop on a small graph, one minibatch per call: launches and host work count, not bandwidth
        {"name": "sage_small", "op": "sage", **small, "batch": 1024, "fanouts": "10,5", "replace": False, "weights": False},
        # the same loop on a large graph, three hops, edge weights carried along into the blocks
        {"name": "sage_products", "op": "sage", **products, "batch": 1024, "fanouts": "15,10,5", "replace": False,
         "weights": True},
        # the throughput form: hundreds of minibatches sampled and relabelled by one call per hop
        {"name": "superbatch_500", "op": "superbatch", **products, "batches": 500, "batch": 1024, "fanouts": "15,10,5",
         "replace": False},
        # the super-batch operators called one by one (fused sample, then per-minibatch relabel), a ragged batch size
        {"name": "superbatch_ops", "op": "superbatch_ops", **products, "batches": 61, "batch": 1000, "fanouts": "10,10",
         "replace": False},
        # layer-wise importance sampling: 2 layers, row probability = sum of squared weights, weighted list sampling
        {"name": "layerwise", "op": "layerwise", **layered, "batch": 512, "layer": 512, "layers": 2},
        # adaptive sampling of a hub-heavy frontier: edge score by SDDMM, softmax per column, weighted sampling
        {"name": "adaptive", "op": "adaptive", **products, "seeds": 2048, "features": 256, "fanout": 10},
        # walks of one training minibatch: a chain of dependent reads, far too few walkers to fill the chip
        {"name": "walk_minibatch", "op": "walk", **products, "walkers": 1024, "length": 80, "sinks": 0.0},
        # walks from every start node of an epoch over a graph far larger than the caches
        {"name": "walk_epoch", "op": "walk", **papers, "walkers": 10_000_000, "length": 80, "sinks": 0.03},
        # a large column slice with edge weights, COO out (the first step of every non-fused sampler)
        {"name": "slice_columns", "op": "slice", **products, "seeds": 262_144, "hubs": False},
        # importance-weighted neighbours of a slice, as blocks
        {"name": "weighted", "op": "weighted", **products, "seeds": 65_537, "fanout": 16, "replace": False},
        # feature rows of a frontier; 100 floats per row, so rows start on 16-byte but not on 128-byte boundaries
        {"name": "gather_features", "op": "gather", "nodes": 2_450_000, "edges": 0, "rows": 1_000_000, "features": 100},
        # the subgraph induced by a neighbourhood (all edges among the given nodes, with their weights)
        {"name": "induced", "op": "induced", **products, "seeds": 20_000},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    op = rng.choice(["sage", "sage", "superbatch", "superbatch", "superbatch_ops", "layerwise", "adaptive", "walk", "slice",
                     "weighted", "gather", "induced"])
    nodes = _log(rng, 50_000, 2_450_000)
    case = {"op": op, "nodes": nodes, "edges": nodes * rng.randint(12, 50)}
    if op == "sage":
        case.update(batch=_log(rng, 64, 8192), fanouts=rng.choice(["10,5", "15,10,5", "25,10", "5,5,5", "20,20"]),
                    replace=rng.random() < 0.2, weights=rng.random() < 0.5)
    elif op == "superbatch":
        case.update(batches=_log(rng, 2, 300), batch=_log(rng, 128, 1024),
                    fanouts=rng.choice(["10,5", "15,10,5", "25,10", "5,5,5"]), replace=rng.random() < 0.2)
    elif op == "superbatch_ops":
        case.update(batches=_log(rng, 2, 200), batch=_log(rng, 128, 1024), fanouts=rng.choice(["10,5", "10,10", "25,10"]),
                    replace=rng.random() < 0.2)
    elif op == "layerwise":
        case.update(batch=_log(rng, 128, 2048), layer=_log(rng, 128, 2048), layers=rng.choice([2, 3]))
    elif op == "adaptive":
        case.update(seeds=_log(rng, 256, 8192), features=rng.choice([64, 100, 128, 256]), fanout=rng.choice([5, 10, 25]))
    elif op == "walk":
        case.update(walkers=_log(rng, 256, 1_000_000), length=rng.randint(5, 100), sinks=rng.choice([0.0, 0.03]))
    elif op == "slice":
        case.update(seeds=min(nodes, _log(rng, 256, 262_144)), hubs=rng.random() < 0.3)
        if case["hubs"]:
            case["seeds"] = min(case["seeds"], 8192)
    elif op == "weighted":
        case.update(seeds=min(nodes // 2, _log(rng, 256, 131_072)), fanout=rng.choice([5, 10, 16, 25, 40]),
                    replace=rng.random() < 0.2)
    elif op == "gather":
        case.update(edges=0, rows=_log(rng, 1000, 2_000_000), features=rng.choice([1, 16, 64, 100, 128, 256, 602]))
    else:
        case.update(seeds=min(nodes // 8, _log(rng, 512, 40_000)))
    return case


# ---- graphs ------------------------------------------------------------------------------------------------------------
# Outputs of another seed have to have the same sizes to be compared, and the size of a sample depends on the graph.  So the
# shape of the graph, of the seed set and of the draws is that of the case, and the seed decides which node gets which id
# (and with it where every column lies, what every table holds and in what order) and all the values: features and carried
# weights.  Walks, whose trace has one size whatever they meet, take graph and starts from the seed.
def _shift(nodes, edges):
    """Rank shift that puts the largest degree near 1.5 * sqrt(edges)."""
    top, shift = 1.5 * math.sqrt(edges), 1.0
    for _ in range(40):
        norm = (nodes + shift) ** 0.25 - shift ** 0.25
        shift = max(1.0, (edges * 0.25 / norm / top) ** (4.0 / 3.0))
    return shift


class _Ids:
    """id = (rank * stride + offset) mod nodes: popularity ranks scattered over the ids, another way for every seed."""

    def __init__(self, nodes, seed):
        pick = random.Random(seed)
        self.nodes, self.offset = nodes, pick.randrange(nodes)
        self.stride = int(nodes * pick.uniform(0.3, 0.7)) | 1
        while math.gcd(self.stride, nodes) != 1:
            self.stride += 2
        self.inverse = pow(self.stride, -1, nodes)

    def of(self, rank):
        return rank.mul(self.stride).add_(self.offset).remainder_(self.nodes)

    def rank_of_all(self):
        return torch.arange(self.nodes, device="cuda").sub_(self.offset).mul_(self.inverse).remainder_(self.nodes)


def _popular(case, count, gen):
    """`count` ranks drawn by popularity."""
    n, shift = case["nodes"], _shift(case["nodes"], case["edges"])
    lo, hi = shift ** 0.25, (n + shift) ** 0.25
    x = torch.rand(count, generator=gen, device="cuda", dtype=torch.float64).mul_(hi - lo).add_(lo)
    return x.square_().square_().sub_(shift).to(torch.int64).clamp_(0, n - 1)


def _graph(case, ids, gen, weighted):
    """(indptr, indices, weights or None) with everything drawn from `gen` but the ids."""
    n, m = case["nodes"], case["edges"]
    shift = _shift(n, m)
    norm = ((n + shift) ** 0.25 - shift ** 0.25) * 4.0
    degree = torch.arange(n, device="cuda").to(torch.float64).add_(shift + 0.5).pow_(-SKEW).mul_(m / norm)
    degree = degree.add_(torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)).to(torch.int64)
    if case.get("sinks", 0.0) > 0:
        degree[torch.rand(n, generator=gen, device="cuda") < case["sinks"]] = 0
    rank = ids.rank_of_all()
    by_id = degree[rank]
    indptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(by_id, 0, out=indptr[1:])
    total = int(indptr[-1])
    if case["op"] == "walk":  # columns in id order as they are drawn: no second copy of the edges
        indices = torch.empty(total, dtype=torch.int64, device="cuda")
        for at in range(0, total, CHUNK):
            part = indices[at:at + CHUNK]
            part.copy_(ids.of(_popular(case, part.numel(), gen)))
        return indptr, indices, None
    by_rank = torch.empty(total, dtype=torch.int64, device="cuda")
    for at in range(0, total, CHUNK):
        part = by_rank[at:at + CHUNK]
        part.copy_(ids.of(_popular(case, part.numel(), gen)))
    first = torch.cumsum(degree, 0).sub_(degree)
    source = torch.repeat_interleave(first[rank] - indptr[:-1], by_id, output_size=total)
    source += torch.arange(total, device="cuda")
    weights = 1.0 - torch.rand(total, generator=gen, device="cuda") if weighted else None  # (0, 1]
    return indptr, by_rank[source], weights[source] if weighted else None


def _uniform_ranks(nodes, count, gen):
    return torch.randperm(nodes, generator=gen, device="cuda")[:count]


def _hub_ranks(case, count, gen):
    """Distinct nodes met in proportion to their popularity, in no order: the frontier of an earlier hop."""
    got = torch.unique(_popular(case, 4 * count + 64, gen))
    while got.numel() < count:
        got = torch.unique(torch.cat([got, _uniform_ranks(case["nodes"], count, gen)]))
    return got[torch.randperm(got.numel(), generator=gen, device="cuda")[:count]]


def prepare(case, seed):
    op, n = case["op"], case["nodes"]
    values, shape = torch.Generator(device="cuda"), torch.Generator(device="cuda")
    values.manual_seed(seed)
    shape.manual_seed(seed + 1 if op == "walk" else SHAPE_SEED)
    state = {"case": case, "fanouts": [int(k) for k in case.get("fanouts", "0").split(",")]}
    if op == "gather":
        state["features"] = torch.randn(n, case["features"], generator=values, device="cuda")
        state["index"] = torch.randint(0, n, (case["rows"],), generator=values, device="cuda")
        return state
    ids = _Ids(n, seed)
    indptr, indices, weights = _graph(case, ids, shape, op in ("weighted", "layerwise"))
    if op in ("slice", "induced") or case.get("weights", False):
        weights = 1.0 - torch.rand(indices.numel(), generator=values, device="cuda")
    state["graph"] = gs.Matrix().load_csc(indptr, indices, weights)
    if op in ("superbatch", "superbatch_ops"):
        # epochs over a training split, shuffled, cut into minibatches of equal size
        split = _uniform_ranks(n, max(case["batch"], int(n * 0.08)), shape)
        per = split.numel() // case["batch"]
        parts = []
        while len(parts) * per < case["batches"]:
            parts.append(split[torch.randperm(split.numel(), generator=shape, device="cuda")][:per * case["batch"]])
        ranks = torch.cat(parts)[:case["batches"] * case["batch"]]
        state["seeds_ptr"] = torch.arange(0, case["batches"] + 1, device="cuda") * case["batch"]
        state["csc"] = (indptr, indices)
    elif op in ("adaptive", "induced") or case.get("hubs", False):
        ranks = _hub_ranks(case, case["seeds"], shape)
    else:
        ranks = _uniform_ranks(n, min(n, case.get("batch") or case.get("walkers") or case["seeds"]), shape)
    state["seeds"] = ids.of(ranks)
    if op == "adaptive":
        state["features"] = torch.randn(n, case["features"], generator=values, device="cuda")
    if op == "layerwise":
        # the rows of a layer are chosen by id, so its size is the seed's: a training step reads it from buffers of one size
        bound, floats = 1 << 19, torch.float32
        state["blocks"] = [[torch.zeros(bound, dtype=t, device="cuda") for t in (torch.int64, torch.int64, torch.int64, floats)]
                           for _ in range(case["layers"])]
    return state


# ---- passes --------------------------------------------------------------------------------------------------------------
def _block(b):
    return [t for t in (b.tensor1, b.tensor2, b.src_ids, b.edge_ids, b.edge_weight) if t is not None] + [b.num_src, b.num_dst]


def _sage(state):
    graph, seeds, out = state["graph"], state["seeds"], []
    for k in state["fanouts"]:
        block = graph.fused_columnwise_slicing_sampling(seeds, k, state["case"]["replace"]).to_block()
        out.append(_block(block))
        seeds = block.src_ids
    return out


def _superbatch(state):
    indptr, indices = state["csc"]
    hops = ops.sage_sample_batches(indptr, indices, state["seeds"], state["seeds_ptr"], state["fanouts"],
                                   replace=state["case"]["replace"])
    keep = ("sub_indptr", "indices", "relabeled", "select_index", "indices_ptr", "frontier", "frontier_ptr")
    return [[hop[key] for key in keep] for hop in hops]


def _superbatch_ops(state):
    indptr, indices = state["csc"]
    seeds, ptr, out = state["seeds"], state["seeds_ptr"], []
    for k in state["fanouts"]:
        sub_indptr, sub_indices, select = ops.fused_csc_col_slicing_sampling(indptr, indices, seeds, k,
                                                                             state["case"]["replace"])
        indices_ptr = ops.batch_edge_offsets(sub_indptr, ptr)
        frontier, frontier_ptr, relabeled, _ = ops.batch_csr_relabel(seeds, ptr, sub_indices, indices_ptr)
        out.append([sub_indptr, sub_indices, select, indices_ptr, frontier, frontier_ptr, relabeled])
        seeds, ptr = frontier, frontier_ptr
    return out


def _layerwise(state):
    graph, seeds, out = state["graph"], state["seeds"], []
    for buffers in state["blocks"]:
        sub = graph[:, seeds]
        prob = sub.sum(1, powk=2)
        selected, _ = gs.list_sampling_with_probs(sub.row_ids(False), prob, state["case"]["layer"], False)
        nodes = torch.cat((seeds, selected)).unique()
        layer = sub[nodes, :].divide(prob[nodes], 1).normalize(0)
        seeds = layer.all_indices()
        block = layer.to_block()
        for buffer, t in zip(buffers, (block.tensor1, block.tensor2, block.src_ids, block.edge_weight)):
            count = min(buffer.numel(), t.numel())
            buffer[:count].copy_(t[:count])
        out.append(buffers + [prob, selected, block.num_src, block.num_dst, int(block.tensor1.numel())])
    return out


def _adaptive(state):
    features, seeds = state["features"], state["seeds"]
    sub = state["graph"][:, seeds]
    score = gs.ops.u_dot_v(sub, features, features[seeds])
    sub.set_data(torch.exp(score.squeeze(-1) * (0.25 / math.sqrt(features.shape[1]))))
    bias = sub.normalize(0).get_data()
    picked = sub.columnwise_sampling(state["case"]["fanout"], replace=False, bias=bias)
    return [bias, picked.row_indices(), picked._graph._CAPI_get_coo_cols(False), picked.get_data()]


def _slice(state):
    sub = state["graph"].columnwise_slicing(state["seeds"])
    return [sub.row_indices(), sub._graph._CAPI_get_coo_cols(False), sub.get_data()]


def _weighted(state):
    sub = state["graph"][:, state["seeds"]]
    return _block(sub.columnwise_sampling(state["case"]["fanout"], state["case"]["replace"], bias=sub.get_data()).to_block())


def _induced(state):
    sub = state["graph"]._graph._CAPI_fusion_slicing(state["seeds"], state["seeds"])
    indptr, indices, _ = sub._CAPI_get_csc()
    return [indptr, indices, sub._CAPI_get_data("default")]


PASSES = {"sage": _sage, "superbatch": _superbatch, "superbatch_ops": _superbatch_ops, "layerwise": _layerwise,
          "adaptive": _adaptive, "slice": _slice, "weighted": _weighted, "induced": _induced,
          "walk": lambda state: state["graph"].random_walk(state["seeds"], state["case"]["length"]),
          "gather": lambda state: ops.gather_rows(state["features"], state["index"])}


def run(state):
    gs.set_seed(DRAW_SEED)  # the stochastic calls of the pass draw from this stream
    return PASSES[state["case"]["op"]](state)


# ---- work and tolerance ----------------------------------------------------------------------------------------------------
def _spectrum(case):
    """Popularity ranks in log-spaced groups: (nodes per group, mean degree, chance of one node to be drawn)."""
    n, m = case["nodes"], case["edges"]
    shift = _shift(n, m)
    edge = np.unique(np.round(np.geomspace(1, n + 1, 4000)).astype(np.int64)) - 1
    size = np.diff(edge).astype(np.float64)
    share = np.diff((edge + shift) ** 0.25) / ((n + shift) ** 0.25 - shift ** 0.25) / size
    return size, m * share, share


def _hop(case, by_uniform, columns, k, replace):
    """(sampled edges, distinct neighbours) of one hop over `columns` columns."""
    size, degree, share = _spectrum(case)
    chance = size / case["nodes"] if by_uniform else size * share
    edges = columns * float(np.sum(chance * (k if replace else np.minimum(degree, k))))
    return edges, float(np.sum(size * -np.expm1(-edges * share)))


def _edges_of(case, columns, hubs):
    """Edges of `columns` whole columns, and the share of all popularity that those columns' nodes hold."""
    size, degree, share = _spectrum(case)
    taken = size * columns / case["nodes"]
    if hubs:
        pool = size * -np.expm1(-(4.0 * columns + 64) * share)  # popular draws, then a random subset of the distinct ones
        taken = pool * min(1.0, columns / max(1.0, pool.sum()))
    return float(np.sum(taken * degree)), float(np.sum(taken * share))


def _sage_bytes(case, groups, columns):
    """Per hop: offsets and ids of the columns, then per edge the id read, and the id, its position and its relabelled id
    written; the frontier written once."""
    total, uniform = 0.0, True
    for k in (int(x) for x in case["fanouts"].split(",")):
        edges, distinct = _hop(case, uniform, columns, k, case["replace"])
        frontier = min(case["nodes"], columns + distinct)
        total += groups * (32.0 * columns + (32.0 if case.get("weights") is None else 24.0) * edges + 8.0 * frontier)
        if case.get("weights"):
            total += groups * 8.0 * edges
        columns, uniform = frontier, False
    return total


def work(case):
    op = case["op"]
    flops = 0.0
    if op == "sage":
        size = _sage_bytes(case, 1, case["batch"])
    elif op in ("superbatch", "superbatch_ops"):
        size = _sage_bytes(case, case["batches"], case["batch"])
    elif op == "layerwise":
        size, columns, hubs = 0.0, case["batch"], False
        for _ in range(case["layers"]):
            edges, _ = _edges_of(case, min(columns, case["nodes"]), hubs)
            size += 32.0 * columns + 12.0 * edges + 4.0 * case["nodes"]  # the columns read once, the row probabilities written
            flops += 2.0 * edges
            columns, hubs = columns + case["layer"], True
    elif op == "adaptive":
        edges, _ = _edges_of(case, case["seeds"], True)
        size = 32.0 * case["seeds"] + edges * (8.0 + 4.0 * case["features"] + 4.0)
        size += case["seeds"] * (4.0 * case["features"] + 20.0 * case["fanout"])
        flops = 2.0 * case["features"] * edges
    elif op == "walk":
        mean = sum((1.0 - case["sinks"]) ** s for s in range(1, case["length"] + 1))  # live steps of a walker
        size = 8.0 * case["walkers"] * (case["length"] + 2) + 24.0 * case["walkers"] * mean
    elif op == "slice":
        edges, _ = _edges_of(case, case["seeds"], case["hubs"])
        size = 32.0 * case["seeds"] + 32.0 * edges  # id and weight read; id, column and weight written
    elif op == "weighted":
        edges, _ = _edges_of(case, case["seeds"], False)
        picked, distinct = _hop(case, True, case["seeds"], case["fanout"], case["replace"])
        size = 32.0 * case["seeds"] + 4.0 * edges + 36.0 * picked + 8.0 * (case["seeds"] + distinct)
    elif op == "gather":
        size = case["rows"] * (8.0 + 8.0 * case["features"])
    else:
        edges, share = _edges_of(case, case["seeds"], True)
        size = 40.0 * case["seeds"] + 8.0 * edges + 16.0 * edges * share
    return {"bytes": size, "flops": flops}


def tolerance(case):
    if case["op"] == "layerwise":
        # sums of up to thousands of fp32 squares, then quotients of them; ids chosen by those may swap at a tie
        return {"rel": 1e-5, "max": 2e-4, "differ": 1e-3}
    if case["op"] == "adaptive":
        # fp32 dot products through exp and a softmax; the choice of a column may swap at a tie
        return {"rel": 1e-5, "max": 2e-4, "differ": 1e-3}
    return "exact"  # ids, offsets and copied values
