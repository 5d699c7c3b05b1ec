"""The work that users of the code generator give it, as cases to time.

Every case goes through a public entry point with the objects that a program keeps
between calls (a generator, a batch compiler, a server) and returns everything the call
produces.  Programs are the seeded synthetic ones of ptilopsis_gb300.synth; sizes are
those of its configurations c0 to c4, of the tests and of the benchmark.

A case's "kind" says which entry point it uses:

  plain    RvGenerator: one program, host arrays in and host words out, or (resident)
           CUDA tensors in and the words left on the device
  batch    BatchCompiler: independent programs in one call
  server   CompileServer: requests of mixed sizes, submitted together
  flatten  flatten: a parser's tree in any node order to post-order arrays

Words, function tables and flattened trees are whole numbers, so exact() has no values.
"""
from __future__ import annotations

import dataclasses
import json
import math
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from ptilopsis_gb300 import DepthTree, RvGenerator, flatten
from ptilopsis_gb300.batch import BatchCompiler, CompileServer
from ptilopsis_gb300.synth import SynthParams, config_params, generate

WORDS_PER_NODE = 0.86       # output words per node of the synthetic programs
BATCH_MEAN_NODES = 69_600   # mean program of the c3 distribution
SMALL_MEAN_NODES = 6_500    # mean of the server's small requests
SERVER_MEAN_NODES = 95_000  # mean of the server's size mix


def listed():
    return [
        # the smallest call: a script of four short functions; launches and syncs count
        _plain("plain_script", functions=4, median=400.0),
        # configuration c0, an ordinary source file: 16 functions, about 20k nodes
        _plain("plain_file", functions=16, median=1250.0),
        # the largest program of the batched configuration, compiled where a GPU flattening
        # left it: device arrays in, words read on the device
        _plain("plain_resident", functions=512, median=890.0, sigma=0.5, nesting=32, resident=True),
        # configuration c1, a large program with deep nesting, a quarter of its functions
        # holding more values than there are registers
        _plain("plain_large", functions=2048, median=1000.0, sigma=1.5, max_fn=7000, nesting=64, spill=0.25),
        # configuration c2 at three tenths of its functions: generated code, deep
        # expressions, half of them float
        _plain("plain_huge", functions=9830, median=1500.0, sigma=1.2, max_fn=4000, nesting=64,
               expr_depth=12, float_frac=0.5),
        # the reference's -s flag on a program of ordinary size and odd function count
        _plain("plain_scalar", functions=167, median=530.0, sigma=0.5, nesting=32, scalar=True),
        # a build of many small files in one call
        _batch("batch_small", "small", 64),
        # the batched configuration (c3), an eighth of its 4,096 uneven programs
        _batch("batch_uneven", "c3", 512),
        # the same distribution with the scalar generator's output
        _batch("batch_scalar", "c3", 128, scalar=True),
        # a burst of compile requests (c4: four fifths small, the rest 100k to 2M nodes)
        {"name": "server_burst", "kind": "server", "requests": 48},
        # a parser's tree on the host, nodes in the order a parallel parser left them
        _flatten("flatten_host", nodes=517995, functions=512, sigma=0.0, resident=False),
        # a large tree already on the device, flattened for a compile there
        _flatten("flatten_resident", nodes=4305469, functions=2048, sigma=0.0, resident=True),
    ]


def _plain(name, functions, median, sigma=0.0, max_fn=0, nesting=8, spill=0.0, expr_depth=6, float_frac=0.3,
           scalar=False, resident=False):
    return {"name": name, "kind": "plain", "functions": functions, "median": median, "sigma": sigma,
            "max_fn": max_fn, "nesting": nesting, "spill": spill, "expr_depth": expr_depth,
            "float_frac": float_frac, "scalar": scalar, "resident": resident}


def _batch(name, preset, programs, scalar=False):
    return {"name": name, "kind": "batch", "preset": preset, "programs": programs, "scalar": scalar}


def _flatten(name, nodes, functions, sigma, resident):
    return {"name": name, "kind": "flatten", "nodes": nodes, "functions": functions, "sigma": sigma,
            "resident": resident}


def _log_between(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """A case of the listed ranges: one program of 100 nodes to 17M, 2 to 400 programs
    in a batch, 3 to 40 requests, a tree of 1k to 4M nodes."""
    kind = rng.choice(["plain", "plain", "plain", "batch", "batch", "server", "flatten"])
    if kind == "plain":
        scalar = rng.random() < 0.25
        functions = round(_log_between(rng, 1, 1200 if scalar else 9000))
        case = _plain("", functions=functions, median=round(_log_between(rng, 100, 1500), 1),
                      sigma=round(rng.uniform(0.0, 1.2), 3), max_fn=rng.randint(2500, 4000),
                      nesting=rng.choice([8, 16, 32, 64]), spill=rng.choice([0.0, 0.0, 0.25]),
                      expr_depth=rng.choice([6, 6, 9, 12]), float_frac=rng.choice([0.0, 0.3, 0.5]),
                      scalar=scalar, resident=rng.random() < 0.3)
    elif kind == "batch":
        scalar = rng.random() < 0.3
        preset = rng.choice(["small", "c3"])
        case = _batch("", preset, round(_log_between(rng, 2, 120 if scalar else 400)), scalar=scalar)
    elif kind == "server":
        case = {"kind": "server", "requests": rng.randint(3, 40)}
    else:
        nodes = round(_log_between(rng, 1000, 4_000_000))
        functions = max(1, round(nodes / rng.uniform(600, 2100)))
        case = _flatten("", nodes=nodes, functions=functions, sigma=0.0, resident=rng.random() < 0.5)
    case.pop("name", None)
    return case


# ---- inputs
def _seed(seed):
    return (0x50544C10 + 7919 * seed) & 0xFFFFFFFF


def _params(case, seed):
    return SynthParams(seed=_seed(seed), n_functions=case["functions"],
                       median_fn_nodes=case["median"], sigma=case["sigma"], max_fn_nodes=case["max_fn"],
                       max_expr_depth=case["expr_depth"], float_frac=case["float_frac"],
                       max_nesting=case["nesting"], spill_frac=case["spill"])


def _generate_all(params):
    with ThreadPoolExecutor(max_workers=min(16, os.cpu_count() or 1)) as pool:
        return list(pool.map(generate, params))


def _small_params(seed, k):
    """A small request: 1k to 10k nodes, as the server's small ones."""
    rng = np.random.default_rng([seed, k])
    total = float(rng.uniform(1000, 10000))
    functions = int(np.clip(total / 800.0, 2, 1024))
    return SynthParams(seed=int(rng.integers(1 << 32)), n_functions=functions, median_fn_nodes=total / functions,
                       sigma=0.6, max_nesting=32)


def _server_params(seed, k):
    """Request k of a burst in the c4 size mix: every fifth one large, so that bursts of
    one length are of about one size."""
    if k % 5 != 2:
        return _small_params(seed, k)
    rng = np.random.default_rng([seed, k])
    total = float(np.clip(np.exp(math.log(300000.0) + 0.8 * rng.standard_normal()), 100000, 2000000))
    functions = int(np.clip(total / 800.0, 2, 1024))
    return SynthParams(seed=int(rng.integers(1 << 32)), n_functions=functions, median_fn_nodes=total / functions,
                       sigma=0.6, max_nesting=32)


def _parser_tree(case, seed):
    """The five arrays of a parser's tree of exactly case["nodes"] nodes, in a random
    order: a program of about nine tenths of them, and empty statements at its root."""
    n = case["nodes"]
    functions = case["functions"]
    tree = generate(SynthParams(seed=_seed(seed), n_functions=functions, median_fn_nodes=0.9 * n / functions,
                                sigma=case["sigma"], max_nesting=32))
    more = n - tree.n
    if more < 0:
        raise ValueError("the program is larger than the case's tree")
    root = tree.n - 1
    children = int((tree.parent == root).sum())
    fill = np.zeros(more, np.uint8)
    type_, rtype = np.concatenate([tree.type, fill]), np.concatenate([tree.rtype, fill])
    parent = np.concatenate([tree.parent, np.full(more, root, np.int32)])
    child_idx = np.concatenate([tree.child_idx, np.arange(children, children + more, dtype=np.int32)])
    data = np.concatenate([tree.data, np.arange(more, dtype=np.uint32)])
    at = np.random.default_rng(seed).permutation(n).astype(np.int32)  # node v goes to at[v]
    parent = np.where(parent >= 0, at[np.maximum(parent, 0)], -1).astype(np.int32)
    out = []
    for a in (type_, rtype, parent, child_idx, data):
        b = np.empty_like(a)
        b[at] = a
        out.append(b)
    return out


# The generators, batch compilers and servers that a program keeps: one per case, made
# with its first inputs and used for all that follow.
_kept = {}


def _keep(case, make):
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "plain":
        tree = generate(_params(case, seed))
        if case["resident"]:
            tree = tree.to("cuda")
            torch.cuda.synchronize()
        gen = _keep(case, lambda: RvGenerator(tree, scalar=case["scalar"]))
        return {"case": case, "gen": gen, "tree": tree, "out": _output(case)}
    if kind == "batch":
        k = case["programs"]
        if case["preset"] == "small":
            params = [_small_params(seed, p) for p in range(k)]
        else:
            params = [config_params("c3", program=4096 * (1 + seed) + p) for p in range(k)]
        trees = _generate_all(params)
        return {"case": case, "compiler": _keep(case, lambda: BatchCompiler(tiles=None, scalar=case["scalar"])),
                "trees": trees, "out": _output(case)}
    if kind == "server":
        trees = _generate_all([_server_params(seed, k) for k in range(case["requests"])])
        return {"case": case, "server": _keep(case, lambda: CompileServer(slots=3)), "trees": trees,
                "out": _output(case)}
    arrays = _parser_tree(case, seed)
    if case["resident"]:
        arrays = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda() for a in arrays]
    return {"case": case, "arrays": arrays}


# ---- passes
class _Output:
    """A program's own buffers for the words and tables of what it compiles, one program
    after the other, zeros behind the last."""

    def __init__(self, words, functions, resident=False):
        self.words = torch.zeros(words, dtype=torch.int32, device="cuda") if resident else np.zeros(words, np.int32)
        self.table = {name: np.zeros(functions, np.int32) for name in ("starts", "ends", "sizes", "ids")}
        self.all = {"words": self.words, **self.table}

    def put(self, compiled):
        """compiled: (words, table) of each program, the words of a resident compile a
        CUDA tensor."""
        w = f = 0
        for words, table in compiled:
            self.words[w:w + len(words)] = words
            w += len(words)
            end = f + len(table["ids"])
            for name, to in self.table.items():
                to[f:end] = table[name].view(np.int32)
            f = end
        return self.all


def _output(case):
    """Room for the words of any seed's programs (under 0.9 words a node, sizes varying
    as _params, config_params and _server_params say)."""
    if case["kind"] == "plain":
        functions = case["functions"]
        words = int(_expected_nodes(case) + 6000 * math.sqrt(functions)) + 4000
        return _Output(words, functions, case["resident"])
    if case["kind"] == "server":
        count = case["requests"]
        return _Output(10_000 * count + 1_850_000 * -(-count // 5), 12 * count + 1024 * -(-count // 5))
    count = case["programs"]
    if case["preset"] == "small":
        return _Output(10_000 * count, 16 * count)
    return _Output(int(80_000 * count + 500_000 * math.sqrt(count)), 512 * count)


class _DeviceWords:
    """Device words as an array that torch takes without a copy."""

    def __init__(self, ptr, count):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (count,), "typestr": "<i4", "version": 3}


def _tree_arrays(tree: DepthTree, order):
    out = {name: getattr(tree, name) for name in ("type", "rtype", "parent", "depth", "child_idx")}
    out["data"] = tree.data.view(np.int32) if isinstance(tree.data, np.ndarray) else tree.data
    out["order"] = order
    out["max_depth"] = tree.max_depth
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "plain":
        gen = state["gen"]
        gen.upload(state["tree"])
        if case["resident"]:
            gen.process(to_host=False)
            words = torch.as_tensor(_DeviceWords(*gen.device_instructions()), device="cuda")
        else:
            gen.process()
            words = gen.get_instructions().view(np.int32)
        return state["out"].put([(words, gen.function_table())])
    if kind == "batch":
        compiler, trees = state["compiler"], state["trees"]
        compiler.compile(trees)
        done = [compiler.result(k) for k in range(len(trees))]
        return state["out"].put([(c.words.view(np.int32), c.table) for c in done])
    if kind == "server":
        server = state["server"]
        tickets = [server.submit(t, copy=False) for t in state["trees"]]
        compiled = [server.result(t) for t in tickets]
        for t in tickets:
            server.release(t)
        return state["out"].put([(c.words.view(np.int32), c.table) for c in compiled])
    return _tree_arrays(*flatten(*state["arrays"]))


# ---- the least that a pass has to move
def _expected_nodes(case):
    kind = case["kind"]
    if kind == "flatten":
        return case["nodes"]
    if kind == "batch":
        return case["programs"] * (SMALL_MEAN_NODES if case["preset"] == "small" else BATCH_MEAN_NODES)
    if kind == "server":
        return case["requests"] * SERVER_MEAN_NODES
    sigma, median, most = case["sigma"], case["median"], case["max_fn"]
    mean = median * math.exp(sigma * sigma / 2.0)
    if most and sigma > 0:  # the mean of a lognormal size cut off at max_fn
        x = math.log(most / median) / sigma
        mean = mean * _normal_cdf(x - sigma) + most * (1.0 - _normal_cdf(x))
    return case["functions"] * mean


def _normal_cdf(x):
    return 0.5 * (1.0 + math.erf(x / math.sqrt(2.0)))


def work(case):
    """Bytes: each tree's 18 bytes a node in and its words out; a flattening reads 14
    bytes a node and writes 22.  The arithmetic is on whole numbers."""
    nodes = _expected_nodes(case)
    if case["kind"] == "flatten":
        return {"bytes": 36.0 * nodes, "flops": 0.0}
    return {"bytes": (18.0 + 4.0 * WORDS_PER_NODE) * nodes, "flops": 0.0}


def exact(case, seed):
    return None
