"""The work that a user of this library has it do, as measurable cases.

A case is a dict of plain values.  `op` says which public entry points one pass takes:

    product        SpmmPlan.run on a plan that is kept (one aggregation of a GNN layer, one run(dim) of the plug-in)
    tiled          TiledSpmmPlan.run: the column-tiled product, for a dense operand larger than L2
    graph_product  a graph that is seen once (a sampled subgraph): degree sort, .block4, spmm() in one go
    setup          what is done once per graph on the device: degree sort with renamed columns, .block4, the plan
    host_setup     the same from and to host arrays, as the file-based workflow has it (degree_sort_files, the .block4 script)
    host_step      HostSpmm.step_batch: the graph and the dense operands from pinned host memory, the results back to it
    host_resident  HostSpmm.run_batch: the graph is on the device, the dense operands come from and go to pinned host memory
    gcn            GcnForward.forward: a two-layer GCN over the whole graph, 128 features

`kind` is the degree distribution: "powerlaw" (symmetric, GCN-normalised, self loops: citation, social and web graphs),
"heavy" (log-normal degrees, hundreds of neighbours per node: protein and similarity graphs), "skewed" (rows only, a few
hub rows that hold a large share of the nonzeros, values uniform).  Sizes are those of the benchmark configurations and
of the tests, and the ranges between them.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "iccad-accel-gcn_b200"))
from accelgcn import degree_sort, gcn, partition, sharded, spmm, synth  # noqa: E402


def listed():
    return [
        # A graph of a few thousand nodes, the narrowest width: one call is launches and latency.
        dict(name="product_tiny", op="product", kind="powerlaw", n=2_048, mean=4, dim=16, relu=False),
        # A citation-sized graph at a width that fills no power of two: still bound by latency.
        dict(name="product_small", op="product", kind="powerlaw", n=16_384, mean=8, dim=60, relu=False),
        # Hub rows of up to 100 000 nonzeros, rows of X that are not 16-byte aligned, the fused activation.
        dict(name="product_skewed", op="product", kind="skewed", n=500_000, mean=30, dim=61, relu=True),
        # Millions of nodes, few neighbours each, X many times larger than L2: bound by HBM.
        dict(name="product_sparse", op="product", kind="powerlaw", n=2_400_000, mean=25, dim=64, relu=False),
        # Hundreds of neighbours per node, X fits L2: bound by the gather from L2.
        dict(name="product_heavy", op="product", kind="heavy", n=250_000, mean=490, dim=64, relu=False),
        # The same graph at the full width: X no longer fits L2, so A is cut into column ranges.
        dict(name="tiled_heavy", op="tiled", kind="heavy", n=250_000, mean=490, dim=128, relu=False),
        # A sampled subgraph that is ordered, partitioned and multiplied once.
        dict(name="graph_product_small", op="graph_product", kind="powerlaw", n=16_384, mean=8, dim=60, relu=False),
        # Set-up of a large graph on the device.
        dict(name="setup_sparse", op="setup", kind="powerlaw", n=2_400_000, mean=25, dim=64, relu=False),
        # The file workflow: arrays read from disk are ordered and partitioned and go back to disk.
        dict(name="host_setup_skewed", op="host_setup", kind="skewed", n=500_000, mean=30, dim=64, relu=False),
        # A harness that keeps everything in host memory and hands the graph over with every step.
        dict(name="host_step_skewed", op="host_step", kind="skewed", n=500_000, mean=30, dim=64, relu=False),
        # A host caller that multiplies new operands by a graph it has set before.
        dict(name="host_resident_medium", op="host_resident", kind="powerlaw", n=100_000, mean=20, dim=64, relu=False),
        # Full-batch inference of a two-layer GCN on a large graph.
        dict(name="gcn_large", op="gcn", kind="powerlaw", n=5_000_000, mean=20, dim=128, relu=True),
    ]


def _between(rng, lo, hi):
    """An integer of [lo, hi], spread over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dim(rng):
    """A width of 16 .. 128: as often a multiple of 4 as any."""
    return 4 * rng.randint(4, 32) if rng.random() < 0.5 else rng.randint(16, 128)


def draw(rng):
    op = rng.choice(["product", "product", "product", "tiled", "graph_product", "setup", "host_setup", "host_step", "host_resident", "gcn"])
    case = dict(op=op, kind="powerlaw", n=0, mean=0, dim=_dim(rng), relu=False)
    if op == "product":
        case["kind"] = rng.choice(["powerlaw", "powerlaw", "skewed", "heavy"])
        case["relu"] = rng.random() < 0.5
        case["n"], case["mean"] = {"powerlaw": lambda: (_between(rng, 2_048, 2_400_000), rng.randint(4, 25)),
                                   "skewed": lambda: (_between(rng, 20_000, 500_000), rng.randint(10, 30)),
                                   "heavy": lambda: (_between(rng, 20_000, 250_000), rng.randint(100, 490))}[case["kind"]]()
    elif op == "tiled":
        case.update(kind="heavy", n=rng.randint(180_000, 250_000), mean=rng.randint(250, 490), dim=4 * rng.randint(28, 32))
    elif op == "graph_product":
        case.update(n=_between(rng, 2_048, 200_000), mean=rng.randint(4, 25))
    elif op == "setup":
        case.update(n=_between(rng, 16_384, 2_400_000), mean=rng.randint(4, 25))
    elif op == "host_setup":
        case.update(kind=rng.choice(["powerlaw", "skewed"]), n=_between(rng, 20_000, 500_000), mean=rng.randint(10, 30))
    elif op == "host_step":
        case.update(kind="skewed", n=_between(rng, 20_000, 500_000), mean=rng.randint(10, 30))
    elif op == "host_resident":
        case.update(n=_between(rng, 16_384, 500_000), mean=rng.randint(8, 25))
    else:
        case.update(n=_between(rng, 16_384, 5_000_000), mean=rng.randint(8, 20), dim=128, relu=True)
    return case


@functools.lru_cache(maxsize=2)
def _weights(n, mean, max_w):
    return synth.power_law_weights(n, 2.2, float(mean), max_w)


def _graph(case, seed):
    """The graph in its own node order, on the GPU.  A case has one degree sequence (so that what the set-up returns has
    one size); the seed names the nodes and, where the values are not those of the normalisation, draws them."""
    n, mean = case["n"], case["mean"]
    if case["kind"] == "powerlaw":
        g = synth.chung_lu("powerlaw", n, _weights(n, mean, min(20_000.0, n / 4)), n * mean, 1, "cuda")
    elif case["kind"] == "heavy":
        g = synth.chung_lu("heavy", n, synth.log_normal_weights(n, 1.0, mean, 1), n * mean, 1, "cuda", self_loops=False)
    else:
        g = synth.skewed_rows("skewed", n, 1.8, max(400, n // 5), n * mean, 1, "cuda")
    name = torch.sort(synth.splitmix64(seed, 2, 0, n, "cuda")).indices
    deg = g.indptr.diff().long()
    keys = torch.repeat_interleave(name, deg) * n + name[g.indices.long()]
    keys, order = torch.sort(keys)
    g.vals = g.vals[order] if case["kind"] != "skewed" else 1.0 - synth.uniform_f32(seed, 5, 0, g.nnz, 0.0, 1.0, "cuda")
    g.indices = (keys % n).int()
    g.indptr[1:] = torch.cumsum(torch.zeros_like(deg).index_copy_(0, name, deg), 0)
    return g


def _host(t):
    return t.cpu().pin_memory()


def prepare(case, seed):
    op, n, dim = case["op"], case["n"], case["dim"]
    g = _graph(case, seed)
    s = {"op": op, "n": n, "relu": case["relu"]}
    if op in ("setup", "graph_product", "host_setup"):
        s.update(indptr=g.indptr, indices=g.indices, vals=g.vals)
        if op == "graph_product":
            s["x"] = synth.features(n, dim, seed, "cuda")
        if op == "host_setup":
            s.update(indptr=g.indptr.cpu().numpy(), indices=g.indices.cpu().numpy(), vals=g.vals.cpu().numpy())
        return s
    _perm, ip, ix, v = degree_sort.degree_sort_device(g.indptr, g.indices, g.vals, relabel_cols=True)
    del g
    x = synth.features(n, dim, seed, "cuda")
    if op == "tiled":
        s.update(plan=spmm.TiledSpmmPlan(ip, ix, v, n, n, dim=dim), x=x, y=torch.empty_like(x))
    elif op == "gcn":
        shard = sharded.ShardedSpmm(ip, ix, v, 0, 1)
        w = [synth.glorot(128, 128, seed, 8 + k, "cuda") for k in range(2)]
        s.update(forward=gcn.GcnForward(shard, w), x=x, y=torch.empty_like(x))
    else:
        block4 = partition.block_level_partition_device(ip)
        if op == "product":
            s.update(plan=spmm.SpmmPlan(block4, ix, n, n), ix=ix, v=v, x=x, y=torch.empty_like(x))
        else:
            # one pass multiplies two operands: the width of the case and half of it
            x2 = synth.features(n, max(16, dim // 2), seed + 1, "cuda")
            s.update(host=spmm.HostSpmm(), block4=_host(block4), ix=_host(ix), v=_host(v), xs=[_host(x2), _host(x)],
                     ys=[torch.empty(t.shape, pin_memory=True) for t in (x2, x)])
            if op == "host_resident":
                s["host"].set_graph(s["block4"], s["ix"], s["v"], n, n)
    return s


def run(s):
    op = s["op"]
    if op == "product":
        s["plan"].run(s["ix"], s["v"], s["x"], s["y"], relu=s["relu"])
        return s["y"]
    if op == "tiled":
        s["plan"].run(s["x"], s["y"])
        return s["y"]
    if op == "gcn":
        return s["forward"].forward(s["x"], out=s["y"])
    if op == "graph_product":
        # columns keep their names: X stays in the caller's order, Y comes in degree order
        perm, ip, ix, v = degree_sort.degree_sort_device(s["indptr"], s["indices"], s["vals"], relabel_cols=False)
        block4 = partition.block_level_partition_device(ip)
        return perm, spmm.spmm(block4, ix, v, s["x"], s["n"])
    if op == "setup":
        perm, ip, ix, v = degree_sort.degree_sort_device(s["indptr"], s["indices"], s["vals"], relabel_cols=True)
        block4 = partition.block_level_partition_device(ip)
        plan = spmm.SpmmPlan(block4, ix, s["n"], s["n"])
        plan.close()
        return perm, ip, ix, v, block4
    if op == "host_setup":
        perm, ip, ix, v = degree_sort.degree_sort(s["indptr"], s["indices"], s["vals"], relabel_cols=True)
        return perm, ip, ix, v, partition.block_level_partition(ip)
    if op == "host_step":
        return s["host"].step_batch(s["block4"], s["ix"], s["v"], s["xs"], s["n"], outs=s["ys"])
    return s["host"].run_batch(s["xs"], outs=s["ys"])


def work(case):
    op, n, dim = case["op"], case["n"], case["dim"]
    nnz = n * case["mean"]
    blocks = 16 * max(n / 12, nnz / 384)
    product, flops = 8 * nnz + blocks + 8 * n * dim, 2 * nnz * dim
    if op in ("product", "tiled"):
        return {"bytes": product, "flops": flops}
    if op == "gcn":
        return {"bytes": 8 * nnz + blocks + 8 * n * 128 + 2 * 4 * 128 * 128, "flops": 2 * (2 * nnz * 128 + 2 * n * 128 * 128)}
    if op == "graph_product":      # the graph in, the order and Y out
        return {"bytes": 8 * nnz + 8 * n + 8 * n * dim, "flops": flops}
    if op in ("setup", "host_setup"):
        return {"bytes": 16 * nnz + 12 * n + blocks, "flops": 0}
    cols = dim + max(16, dim // 2)
    graph = 8 * nnz + blocks if op == "host_step" else 0
    return {"bytes": graph + 8 * n * cols, "flops": 2 * nnz * cols}


def tolerance(case):
    if case["op"] in ("setup", "host_setup"):
        return "exact"             # whole numbers, and values that are only moved
    if case["op"] == "gcn":
        return {"rel": 1e-3}       # operands of the dense transforms in TF32: 2^-11 each, two layers
    return {"rel": 1e-5}           # fp32 sums, the order of the additions is free
