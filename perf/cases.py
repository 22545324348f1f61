"""The framework's work, as cases a timing program can run.

A case is a dict of plain values.  `prepare` makes what a user's program holds before
the call (graphs from this library's seeded generators, prepared problems, handles on
the GPU), `run` makes one pass through the public entry points and returns its whole
outputs, `work` gives the bytes a pass cannot do without, and `exact` the outputs that
are computed floating-point numbers, in 64 bits.

Kinds of case:
  solve     the de Pina main loop on a handle: Solver reset + run + results ("run"), the
            same as a CUDA graph ("graph"), the per-iteration form ("plain"), or from
            host buffers ("upload": upload + run + results)
  batch     many graphs (or the biconnected components of one) in one launch:
            BatchSolver run + results
  generate  the candidates of a graph on the device: every root's shortest-path tree,
            the candidate test, and the sorted coordinate lists
  labels    the reference GPU layer's call: labels of every tree for one support vector,
            into device memory ("device") or the host's rows ("host")
  forward   the learned proposal's scores of a candidate list
  gradients the proposal's training step up to its gradients
"""
import ctypes
import math

import numpy as np
import torch

from minimumcyclebasis_gb300 import (BatchSolver, GpuStruct, Problem, Solver, batch_graphs, bcc_split,
                                     block_tree_graph, grid_graph, planar_chain_graph, prepare_many, random_graph,
                                     rgg_graph)
from minimumcyclebasis_gb300._native import check_gpu, gpu_lib
from minimumcyclebasis_gb300.devprep import GpuGen, generate_candidates, prepare_on_device
from minimumcyclebasis_gb300.learned import ProposalNet, init_params


def listed():
    return [
        # the first configuration: a 32 x 32 grid, N = 961; a service solving small graphs, bound by latency
        {"name": "solve_grid_32", "kind": "solve", "form": "run", "graph": "grid", "n": 32},
        # the per-iteration form, the shape of the reference's own loop, on an ordinary random graph
        {"name": "plain_random_2k", "kind": "solve", "form": "plain", "graph": "random", "n": 2000},
        # a random geometric graph from host buffers to the basis: upload, solve, results
        {"name": "upload_rgg_10k", "kind": "solve", "form": "upload", "graph": "rgg", "n": 10000},
        # a road-like graph with degree-two chains, solved over and over: the CUDA-graph form
        {"name": "graph_planar_100k", "kind": "solve", "form": "graph", "graph": "planar", "n": 100000},
        # the second configuration: 50k vertices, 100k edges, 29.6M candidates
        {"name": "solve_random_50k", "kind": "solve", "form": "run", "graph": "random", "n": 50000},
        # the biconnected components of one graph (50-150 vertices each), one launch
        {"name": "batch_components_1000", "kind": "batch", "graph": "blocks", "count": 1000, "nmax": 150},
        # many graphs of 50-5000 vertices, one launch
        {"name": "batch_graphs_384", "kind": "batch", "graph": "random", "count": 384, "nmax": 5000},
        # candidate generation, distances in shared memory (up to 53,248 vertices)
        {"name": "generate_random_20k", "kind": "generate", "graph": "random", "n": 20000},
        # candidate generation, distances in global memory
        {"name": "generate_planar_65k", "kind": "generate", "graph": "planar", "n": 65000},
        # the reference GPU layer's label pass over every tree, for one support vector
        {"name": "labels_random_8k", "kind": "labels", "form": "device", "graph": "random", "n": 8000},
        # the proposal's scores of every candidate of the 1M-vertex graph
        {"name": "forward_8m", "kind": "forward", "count": 8437310},
        # one training batch of the proposal (the trainer's default size)
        {"name": "gradients_16k", "kind": "gradients", "count": 16384},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve"] * 4 + ["batch"] * 2 + ["generate"] * 2 + ["labels", "forward", "gradients"])
    if kind == "solve":
        form = rng.choice(["run", "run", "graph", "upload", "plain"])
        graph = rng.choice(["grid", "random", "rgg", "planar"])
        hi = {"grid": 110, "random": 40000, "rgg": 12000, "planar": 80000}[graph]
        lo = {"grid": 8, "random": 300, "rgg": 500, "planar": 1000}[graph]
        if form in ("plain", "upload"):  # one launch pair per iteration; lists made on the host
            hi = {"grid": 70, "random": 8000, "rgg": 8000, "planar": 10000}[graph]
        return {"kind": kind, "form": form, "graph": graph, "n": _log(rng, lo, hi)}
    if kind == "batch":
        if rng.random() < 0.4:
            return {"kind": kind, "graph": "blocks", "count": _log(rng, 100, 1500), "nmax": rng.randint(100, 300)}
        return {"kind": kind, "graph": "random", "count": _log(rng, 16, 384), "nmax": _log(rng, 300, 5000)}
    if kind == "generate":
        graph = rng.choice(["random", "planar", "grid"])
        lo, hi = {"random": (500, 30000), "planar": (1000, 60000), "grid": (20, 150)}[graph]
        return {"kind": kind, "graph": graph, "n": _log(rng, lo, hi)}
    if kind == "labels":
        form = rng.choice(["device", "host"])
        return {"kind": kind, "form": form, "graph": rng.choice(["random", "planar"]),
                "n": _log(rng, 300, 9000 if form == "device" else 3000)}
    if kind == "forward":
        return {"kind": kind, "count": _log(rng, 5000, 8000000)}
    return {"kind": kind, "count": _log(rng, 500, 100000)}


def _graph(case, seed):
    n = case["n"]
    if case["graph"] == "grid":
        return grid_graph(n, n, 1, 100, seed)
    if case["graph"] == "random":
        return random_graph(n, 2 * n, 1, 1000, seed)
    if case["graph"] == "rgg":
        return rgg_graph(n, 4, seed)
    return planar_chain_graph(n, seed=seed)


# Sizes of a family's problem at n, from the generators' graphs: (N, F, n', slots, K, nnz).
# A graph of another seed differs by a few percent.
def _sizes(graph, n):
    if graph == "grid":
        N = (n - 1) ** 2
        return N, 0.33 * n * n, n * n, 4.0 * n * n, 6145 * (N / 961) ** 1.37, 87102 * (N / 961) ** 1.89
    if graph == "random":
        return n + 1, 0.235 * n, 0.83 * n, 3.66 * n, 63285 * (n / 2000) ** 1.91, 547447 * (n / 2000) ** 2.04
    if graph == "rgg":
        return 1.43 * n, 0.433 * n, n, 4.86 * n, 56621 * (n / 1e4) ** 1.1, 767334 * (n / 1e4) ** 1.6
    return 1.08 * n, 0.3 * n, 0.917 * n, 4.0 * n, 208873 * (n / 2e4) ** 1.43, 12109132 * (n / 2e4) ** 1.97


def work(case):
    kind = case["kind"]
    if kind == "solve":  # weights, offsets and lists read; support vectors (lower triangle) and ranks written
        N, _, _, _, K, nnz = _sizes(case["graph"], case["n"])
        return {"bytes": 12 * K + 4 * nnz + N * N / 16 + 8 * N, "flops": 0}
    if kind == "batch":
        if case["graph"] == "blocks":
            s = case["nmax"] / 150
            N, K, nnz = 84 * s, 368 * s ** 1.6, 1742 * s ** 1.9
        else:
            s = case["nmax"] / 5000
            N, K, nnz = 920 * s ** 0.85, 40000 * s ** 1.7, 366000 * s ** 1.9
        return {"bytes": case["count"] * (12 * K + 4 * nnz + N * N / 10 + 8 * N), "flops": 0}
    if kind == "generate":  # pairs, weights, offsets and lists written; one addition per root and slot
        _, F, _, slots, K, nnz = _sizes(case["graph"], case["n"])
        return {"bytes": 16 * K + 4 * nnz + 24 * slots, "flops": F * slots}
    if kind == "labels":  # edge offset and parent read, label written, per tree and position
        _, F, nn, _, _, _ = _sizes(case["graph"], case["n"])
        return {"bytes": 12 * F * nn, "flops": 0}
    rows = case["count"]
    if kind == "forward":
        return {"bytes": 36 * rows, "flops": 2 * rows * 64 * 17}
    return {"bytes": 33 * rows, "flops": 2 * 3 * rows * 64 * 17}


def _room(count):
    """Entries a program reserves for an output whose length the graph decides."""
    return int(2.2 * count) + 4096


def _fill(buffer, values):
    """The caller's output array with `values` at its front (its rest stays as it was)."""
    buffer[:len(values)] = values
    return buffer


def _pinned(a):
    t = torch.empty(a.shape, dtype={"int32": torch.int32, "int64": torch.int64}[a.dtype.name], pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def _features(count, seed):
    """Candidate features as the walk computes them: weight over the median, distance
    and edge shares, log hop counts, rank quantile, log degrees, a constant, padding."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    u = torch.rand((count, 8), device="cuda", generator=g)
    x = torch.zeros((count, 16), device="cuda")
    we = 0.02 + 0.2 * u[:, 0]
    da = (1 - we) * (0.25 + 0.25 * u[:, 1])
    x[:, 0] = torch.exp(1.2 * (2 * u[:, 2] - 1))
    x[:, 1], x[:, 2], x[:, 3] = da, 1 - we - da, we
    ha, hb = torch.floor(2 + 60 * u[:, 3]), torch.floor(2 + 60 * u[:, 4])
    x[:, 4] = torch.log2(1 + ha + hb) / 8
    x[:, 5] = torch.log2(1 + torch.floor((ha + hb) * u[:, 5])) / 8
    x[:, 6] = torch.arange(count, device="cuda") / count
    x[:, 7] = torch.log2(4 + torch.floor(3 * u[:, 6])) / 4
    x[:, 8] = torch.log2(7 + torch.floor(5 * u[:, 7])) / 4
    x[:, 9] = (ha - hb).abs() / (1 + ha + hb)
    x[:, 10] = 1
    y = (torch.rand(count, device="cuda", generator=g) < 0.25 * torch.exp(-3 * x[:, 6])).to(torch.uint8)
    return x.to(torch.bfloat16), y


def _nonzero(seed):
    return seed % (1 << 30) + 1


def prepare(case, seed):
    kind, seed = case["kind"], _nonzero(seed)
    if kind == "solve":
        g = _graph(case, seed)
        # a k-nearest-neighbour graph's edge count, and with it N, is the seed's
        out = np.full(_room(1.43 * case["n"]), -1, np.int64) if case["graph"] == "rgg" else None
        if case["form"] != "upload":
            return {"kind": kind, "form": case["form"], "solver": prepare_on_device(g).solver, "out": out}
        p = Problem.from_graph(g).prepare()
        w = p.candidates()[2]
        off, co = p.cycle_lists()
        return {"kind": kind, "form": "upload", "solver": Solver(p.N, w, off, co), "out": out,
                "lists": (_pinned(w), _pinned(off), _pinned(co))}
    if kind == "batch":
        if case["graph"] == "blocks":
            gs = bcc_split(block_tree_graph(case["count"], nmax=case["nmax"], seed=seed))
        else:
            gs = batch_graphs(case["count"], nmax=case["nmax"], seed=seed)
        ps = prepare_many([Problem.from_graph(g) for g in gs])
        ps = [p for p in ps if not p.info.single_cycle and p.N > 0]
        # the number of selections is the seed's: at most the edges of the largest graphs
        most = case["count"] * (case["nmax"] * 5 // 2)
        return {"kind": kind, "batch": BatchSolver.from_problems(ps), "selected": np.full(most, -1, np.int64),
                "totals": np.full(case["count"], -1, np.int64)}
    if kind == "generate":
        p = Problem.from_graph(_graph(case, seed)).prepare(structure_only=True)
        gen = GpuGen(p)
        # the rank order of the candidates (the host's step between the device's two)
        offs, pairs, weights, _, _ = generate_candidates(p, gen)
        p.rank_candidates(offs, pairs, weights)
        _, edge, w, tree = p.candidates()
        gen.close()
        _, F, _, _, K, nnz = _sizes(case["graph"], case["n"])
        host = [np.full(_room(c), 0, t) for c, t in ((F, np.int64), (K, np.int32), (K, np.int32))]
        dev = [torch.full((_room(c),), -1, dtype=t, device="cuda") for c, t in ((K, torch.int64), (nnz, torch.int32))]
        return {"kind": kind, "problem": p, "gen": GpuGen(p), "ranked": (tree, edge, w), "host": host, "device": dev}
    if kind == "labels":
        p = Problem.from_graph(_graph(case, seed)).prepare(cycle_lists=False, ref_layout=True)
        _, ec = p.coords()
        lv, pp, eo, _ = p.ref_layout()
        rng = np.random.default_rng(seed)
        S = rng.integers(0, 2 ** 63, size=(p.N + 63) // 64 + 1, dtype=np.int64).astype(np.uint64)
        S = S[:(p.N + 63) // 64]
        if p.N % 64:
            S[-1] &= np.uint64((1 << (p.N % 64)) - 1)
        _, F, n, _, _, _ = _sizes(case["graph"], case["n"])  # of this family and size; the seed's differ a little
        if case["form"] == "host":
            gs = GpuStruct(len(ec), p.N, p.n, p.F)
            gs.initialize_memory(ec, lv, pp, eo)
            return {"kind": kind, "form": "host", "struct": gs, "S": S, "labels": np.full(_room(F * n), 2, np.int32)}
        dev = [torch.from_numpy(a.view(t)).cuda() for a, t in ((lv, np.int32), (pp, np.int32), (eo, np.int32),
                                                              (ec, np.int32), (S, np.int64))]
        return {"kind": kind, "form": "device", "arrays": dev, "sizes": (len(ec), p.N, p.F, p.n),
                "labels": torch.full((_room(F * n),), 2, dtype=torch.int32, device="cuda")}
    x, y = _features(case["count"], seed)
    return {"kind": kind, "net": ProposalNet(seed=seed), "x": x, "y": y}


class _Device:
    """A device array of the library seen through the CUDA array interface."""

    def __init__(self, address, count, typestr):
        self.__cuda_array_interface__ = {"data": (address, False), "shape": (count,), "typestr": typestr,
                                         "strides": None, "version": 2}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        s, form = state["solver"], state["form"]
        if form == "upload":
            w, off, co = state["lists"]
            s.upload(weight=w, offsets=off, coords=co)
            s.run()
        elif form == "graph":
            s.run_graph()
        else:
            s.reset()
            if form == "plain":
                s.run_plain()
            else:
                s.run()
        sel, total = s.results()
        return {"selected": sel if state["out"] is None else _fill(state["out"], sel), "total": total}
    if kind == "batch":
        b = state["batch"]
        b.run()
        sel, total = b.results()
        np.concatenate(sel, out=state["selected"][:int(b.N.sum())])
        return {"selected": state["selected"], "totals": _fill(state["totals"], total)}
    if kind == "generate":
        gen = state["gen"]
        offs, pairs, weights, _, _ = generate_candidates(state["problem"], gen)
        nnz = gen.lists(*state["ranked"])
        _, off, co = gen.device_lists()
        host, dev = state["host"], state["device"]
        return {"offsets": _fill(host[0], offs), "pairs": _fill(host[1], pairs), "weights": _fill(host[2], weights),
                "list_offsets": _fill(dev[0], torch.as_tensor(_Device(off, gen.K + 1, "<i8"), device="cuda")),
                "lists": _fill(dev[1], torch.as_tensor(_Device(co, nnz, "<i4"), device="cuda"))}
    if kind == "labels":
        if state["form"] == "host":
            gs = state["struct"]
            gs.copy_support_vector(state["S"])
            return _fill(state["labels"], gs.process_shortest_path()[0].reshape(-1))
        lv, pp, eo, ec, S = (ctypes.c_void_p(t.data_ptr()) for t in state["arrays"])
        edges, N, F, n = state["sizes"]
        check_gpu(gpu_lib().mcbgpu_label_forest_noalloc(lv, pp, eo, ec, edges, S, N, F, n,
                                                        ctypes.c_void_p(state["labels"].data_ptr()), None),
                  "mcbgpu_label_forest_noalloc")
        return state["labels"]
    if kind == "forward":
        return state["net"].forward(state["x"])
    loss, grads = state["net"].gradients(state["x"], state["y"], pos_weight=4.0)
    return {"loss": loss, "grads": grads}


def _params64(seed):
    """The network's parameters as its forward pass takes them: W1 and w2 rounded to
    bfloat16, the biases as they are."""
    p = torch.from_numpy(init_params(_nonzero(seed)))
    w1 = p[:1024].to(torch.bfloat16).double().reshape(64, 16).cuda()
    w2 = p[1088:1152].to(torch.bfloat16).double().cuda()
    return w1, p[1024:1088].double().cuda(), w2, p[1152].double().cuda()


def exact(case, seed):
    if case["kind"] not in ("forward", "gradients"):
        return None  # whole numbers only
    x, y = _features(case["count"], _nonzero(seed))
    w1, b1, w2, b2 = _params64(seed)
    if case["kind"] == "forward":
        return torch.cat([torch.relu(c.double() @ w1.T + b1) @ w2 + b2 for c in x.split(1 << 20)])
    x, y = x.double(), y.double()
    h = torch.relu(x @ w1.T + b1)
    z = h @ w2 + b2
    wt = torch.where(y > 0, 4.0, 1.0).double() / case["count"]
    loss = (wt * torch.nn.functional.softplus(torch.where(y > 0, -z, z))).sum()
    dz = (torch.sigmoid(z) - y) * wt
    dh = torch.where(h > 0, dz[:, None] * w2, torch.zeros_like(h))
    grads = torch.cat([(dh.T @ x).reshape(-1), dh.sum(0), dz @ h, dz.sum().reshape(1)])
    return {"loss": float(loss), "grads": grads.cpu().numpy()}
