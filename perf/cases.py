"""What is measured: products with a GRG through the package's public calls.

A program that uses this package loads one GRG, keeps it resident on the GPU and multiplies many
inputs with it: the graph handle is kept, the inputs are new.  The graphs are the seeded
window-tree graphs of this repository's tests and benchmark, from N=1,000 haplotypes and M=10,000
variants up to N=200,000 and M=250,000 (5e8 edges); a graph is made once per (N, M) and kept, the
last few of them.
"""
from __future__ import annotations

import math
from collections import OrderedDict

import numpy as np
import torch

import grgl_gb300 as gx

WINDOW = 100  # variants per window of the generator
GRAPH_SEED = 42
N_RANGE, M_RANGE, K_MAX = (1_000, 200_000), (3_000, 250_000), 128
LARGEST = 200_000 * 250_000 // WINDOW * 64 * 8  # edge * column * bytes of the costliest listed case

_graphs: "OrderedDict[tuple, gx.GRG]" = OrderedDict()


def _graph(case) -> gx.GRG:
    """The resident graph a program keeps.  With "missing", every tenth variant has a node that
    stands for the samples whose call is missing."""
    key = (case["N"], case["M"], bool(case.get("missing")))
    if key not in _graphs:
        while len(_graphs) >= 3:
            _graphs.popitem(last=False)
        g = gx.window_tree_grg(case["N"], case["M"], seed=GRAPH_SEED)
        if case.get("missing"):
            a = g.export_arrays()
            miss = np.full(g.num_mutations, gx.INVALID_NODE, dtype=np.uint32)
            some = np.random.default_rng(GRAPH_SEED).integers(0, g.num_nodes, size=len(miss[::10]))
            miss[::10] = some
            g = gx.from_csr(g.num_samples, g.ploidy, a["down_off"], a["down_adj"], a["mut_node"], miss_node=miss)
            g.case_miss_node = miss
        _graphs[key] = g.upload()
    _graphs.move_to_end(key)
    return _graphs[key]


def listed():
    return [
        # Allele counts of one small cohort (the size of the recorded fixture graph): a host array
        # in, a host array out, the shortest call there is.
        dict(name="counts small host", op="matmul", N=1_000, M=10_000, K=1, dtype="int32", up=True, host=True),
        # One polygenic score per haplotype on the same cohort, float64 on host arrays.
        dict(name="score small host", op="dot", N=1_000, M=10_000, K=1, dtype="float64", up=False, host=True),
        # Missing calls and diploid inputs on a medium cohort: UP per individual, the missing
        # part in its own output.
        dict(name="missing by individual", op="matmul", N=20_000, M=20_000, K=5, dtype="float64", up=True,
             host=False, missing=True, by_individual=True),
        # One iteration of a PCA by subspace iteration (V Z Z^T with the standardized genotypes).
        dict(name="pca step", op="gram", N=20_000, M=50_000, K=20, dtype="float64", up=True, host=False),
        # Requests of several users on one graph, run as shared traversals.
        dict(name="batch of requests", op="batch", N=50_000, M=50_000, K=24, dtype="float32", up=True, host=False),
        # A phenotype vector against every variant of a large cohort (association scan), float32.
        dict(name="scan K=1 up", op="matmul", N=200_000, M=250_000, K=1, dtype="float32", up=True, host=False),
        # Per-haplotype counts of a marked variant set, the narrowest DOWN product.
        dict(name="burden K=1 down", op="matmul", N=200_000, M=250_000, K=1, dtype="int32", up=False, host=False),
        # Several scores at once, an odd number of them, on host arrays as the reference is called.
        dict(name="scores K=9 host", op="matmul", N=200_000, M=250_000, K=9, dtype="float32", up=False, host=True),
        # Integer counts over many sample groups.
        dict(name="group counts K=48 up", op="matmul", N=200_000, M=250_000, K=48, dtype="int32", up=True,
             host=False),
        # A block of a randomised PCA, one half of an iteration each way.
        dict(name="block K=64 down", op="matmul", N=200_000, M=250_000, K=64, dtype="float32", up=False, host=False),
        dict(name="block K=32 up f64", op="matmul", N=200_000, M=250_000, K=32, dtype="float64", up=True, host=False),
        dict(name="block K=64 down f64", op="matmul", N=200_000, M=250_000, K=64, dtype="float64", up=False,
             host=False),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """A product of any kind on a graph of any size of the ranges, within the largest listed cost."""
    while True:
        N, M = _log_int(rng, *N_RANGE) // 2 * 2, _log_int(rng, *M_RANGE)
        K = _log_int(rng, 1, K_MAX)
        op = rng.choice(["matmul"] * 6 + ["gram", "standardized", "batch", "dot"])
        dtype = rng.choice(["float32", "float64"] if op in ("gram", "standardized", "dot") else
                           ["float32", "float64"] * 2 + ["int32", "int64", "int8", "bool"])
        if op == "batch":
            dtype = "float32"
        case = dict(op=op, N=N, M=M, K=1 if op == "dot" else K, dtype=dtype, up=rng.random() < 0.5,
                    host=op == "dot" or (op == "matmul" and rng.random() < 0.3))
        if op == "matmul" and dtype != "bool" and rng.random() < 0.25:
            option = rng.choice(["by_individual", "missing", "emit_all", "init_vector"])
            if not (option == "emit_all" and N * M > 10**9):
                case[option] = True
        if _edges(case) * _columns(case) * _itemsize(case) <= LARGEST:
            return case


# ---- sizes ----------------------------------------------------------------------------------------


def _edges(case):
    """Nearly every haplotype has one parent per window."""
    return case["N"] * -(-case["M"] // WINDOW)


def _itemsize(case):
    return 1 if case["dtype"] == "bool" else np.dtype(case["dtype"]).itemsize


def _requests(case):
    """(rows, up, standardized) of the batch's requests: narrow and wide ones in both directions."""
    out, left, k = [], case["K"], 0
    while left > 0:
        rows = min(left, (1, 3, 2, 8)[k % 4])
        out.append((rows, k % 2 == 0, k % 3 == 2))
        left -= rows
        k += 1
    return out


def _columns(case):
    return case["K"] * (2 if case["op"] == "gram" else 1)


def work(case):
    """The edges once, one byte each (fewer than 256 nodes of a window can be a haplotype's
    parent), the input once, the output once; an addition per edge and column."""
    N, M, s = case["N"], case["M"], _itemsize(case)
    ins, outs = (N, M) if case["up"] else (M, N)
    if case["op"] == "gram":
        outs = ins
    if case.get("by_individual"):
        ins, outs = (N // 2, M) if case["up"] else (M, N // 2)
    rows = case["K"]
    return {"bytes": _edges(case) * (2 if case["op"] == "gram" else 1) + rows * (ins + outs) * s,
            "flops": _edges(case) * _columns(case)}


# ---- inputs ---------------------------------------------------------------------------------------


def _values(case, shape, gen):
    """Genotype counts for integers, marks for bool, normal deviates for floats."""
    dt = getattr(torch, case["dtype"])
    if case["dtype"] == "bool":
        return torch.rand(shape, generator=gen, device="cuda") < 0.5
    if dt.is_floating_point:
        return torch.randn(shape, generator=gen, device="cuda", dtype=dt)
    return torch.randint(0, 3, shape, generator=gen, device="cuda", dtype=dt)


def prepare(case, seed):
    g = _graph(case)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    op, K, up = case["op"], case["K"], case["up"]
    samples = g.num_individuals if case.get("by_individual") else g.num_samples
    state = {"case": case, "g": g, "direction": gx.UP if up else gx.DOWN}
    if op == "batch":
        state["requests"] = [(_values(case, (rows, g.num_samples if u else g.num_mutations), gen),
                              gx.UP if u else gx.DOWN, std) for rows, u, std in _requests(case)]
        return state
    x = _values(case, (K, samples if up else g.num_mutations), gen)
    kw = {}
    if case.get("by_individual"):
        kw["by_individual"] = True
    if case.get("emit_all"):
        kw["emit_all_nodes"] = True
    if case.get("init_vector"):
        kw["init"] = _values(case, (K,), gen)
    if case.get("missing"):
        kw["miss"] = torch.zeros((K, g.num_mutations), dtype=x.dtype, device="cuda") if up else \
            _values(case, (K, g.num_mutations), gen)
    if case["host"]:
        x = x.cpu().numpy()
        kw = {k: v.cpu().numpy() if isinstance(v, torch.Tensor) else v for k, v in kw.items()}
    if op == "dot":
        x = x[0]
    state.update(x=x, kw=kw)
    return state


def run(state):
    op, g, d = state["case"]["op"], state["g"], state["direction"]
    if op == "batch":
        return gx.matmul_batch(g, state["requests"])
    x, kw = state["x"], state["kw"]
    if op == "dot":
        return gx.dot_product(g, x, d)
    if op == "gram":
        return gx.matmul_gram(g, x, d, standardized=True)
    if op == "standardized":
        return gx.matmul_standardized(g, x, d)
    if "miss" in kw and d == gx.UP:
        kw["miss"][...] = 0  # an UP product adds the missing part to it
        return gx.matmul(g, x, d, **kw), kw["miss"]
    return gx.matmul(g, x, d, **kw)


# ---- the same in 64 bits, by plain torch -----------------------------------------------------------


class _Plain:
    """The graph's edges on the GPU, the haplotypes' apart from the few between inner nodes, and
    the products in the input's 64-bit type."""

    CHUNK = 1 << 29  # values gathered at a time

    def __init__(self, g):
        a = g.export_arrays()
        self.n, self.N = g.num_nodes, g.num_samples
        off = torch.from_numpy(a["down_off"].astype(np.int64)).cuda()
        child = torch.from_numpy(a["down_adj"].view(np.int32)).cuda()
        parent = torch.repeat_interleave(torch.arange(self.n, dtype=torch.int32, device="cuda"), off[1:] - off[:-1])
        leaf = child < self.N
        self.low = child[leaf], parent[leaf]
        pi, ci = parent[~leaf].long(), child[~leaf].long()
        height = torch.ones(self.n, dtype=torch.int64, device="cuda")
        while True:
            h = height.scatter_reduce(0, pi, height[ci] + 1, "amax")
            if torch.equal(h, height):
                break
            height = h
        self.inner = [(ci[height[pi] == h], pi[height[pi] == h]) for h in range(2, int(height.max()) + 1)]
        mut = torch.from_numpy(a["mut_node"].astype(np.int64)).cuda()
        self.mut, self.has_mut = mut.clamp(max=self.n - 1), mut < self.n
        miss = getattr(g, "case_miss_node", None)
        if miss is not None:
            miss = torch.from_numpy(miss.astype(np.int64)).cuda()
            self.miss, self.has_miss = miss.clamp(max=self.n - 1), miss < self.n

    def _along(self, val, src, dst):
        step = max(1, self.CHUNK // val.shape[1])
        for b in range(0, len(src), step):
            val.index_add_(0, dst[b:b + step].long(), val[src[b:b + step].long()])

    def up(self, val):
        self._along(val, *self.low)
        for child, parent in self.inner:
            self._along(val, child, parent)
        return val

    def down(self, val):
        for child, parent in reversed(self.inner):
            self._along(val, parent, child)
        self._along(val, self.low[1], self.low[0])
        return val

    def product(self, x, up, case, init=None, miss=None):
        """K x columns in, K x columns out (and the missing part of an UP product)."""
        K, ploid = x.shape[0], 2 if case.get("by_individual") else 1
        val = torch.zeros((self.n, K), dtype=x.dtype, device="cuda")
        if init is not None:
            val += init
        if up:
            val[:self.N] += x.t().repeat_interleave(ploid, 0)
            self.up(val)
        else:
            val.index_add_(0, self.mut[self.has_mut], x.t()[self.has_mut])
            if miss is not None:
                val.index_add_(0, self.miss[self.has_miss], miss.t()[self.has_miss])
            self.down(val)
        if case.get("emit_all"):
            return val.t()
        if not up:
            return val[:self.N].reshape(self.N // ploid, ploid, K).sum(1).t()
        out = val[self.mut].t() * self.has_mut
        return (out, val[self.miss].t() * self.has_miss) if miss is not None else out

    def standardized(self, x, up):
        count = self.product(torch.ones((1, self.N), dtype=torch.float64, device="cuda"), True, {})[0]
        p = count / self.N
        inv = torch.where(p * (1 - p) > 0, 1 / (p * (1 - p)).clamp(min=1e-300).sqrt(), torch.zeros_like(p))
        if up:
            return (self.product(x, True, {}) - x.sum(1, keepdim=True) * p) * inv
        w = x * inv
        return self.product(w, False, {}) - (w @ p)[:, None]


def exact(case, seed):
    state = prepare(case, seed)
    plain = _Plain(state["g"])

    def wide(v):
        v = torch.as_tensor(v).cuda()
        return v.double() if v.is_floating_point() else v.long()

    def narrow(v):
        if case["dtype"] == "bool":
            return v % 2 == 1
        return v if case["dtype"].startswith("float") else v.to(getattr(torch, case["dtype"]))

    up, op = case["up"], case["op"]
    if op == "batch":
        return [plain.standardized(wide(x), d == gx.UP) if std else
                plain.product(wide(x), d == gx.UP, {}) for x, d, std in state["requests"]]
    x, kw = wide(state["x"]), state["kw"]
    if op == "dot":
        return plain.product(x[None], up, {})[0]
    if op == "standardized":
        return plain.standardized(x, up)
    if op == "gram":
        return plain.standardized(plain.standardized(x, up), not up)
    init = wide(kw["init"]) if "init" in kw else None
    got = plain.product(x, up, case, init, wide(kw["miss"]) if "miss" in kw else None)
    return tuple(narrow(v) for v in got) if isinstance(got, tuple) else narrow(got)
