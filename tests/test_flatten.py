"""AST flattening: a parent-pointer tree in any node order into the reference's DepthTree
(pareas-ast/src/codegen/depthtree.cpp:11-100).  The oracle's restatement is pinned
against the reference's own DepthTree constructor (built from its sources) and against
the post-order trees the generator tests use; the GPU (ptl_flatten) is checked against
the oracle on shuffled trees, degenerate shapes and malformed inputs."""
from __future__ import annotations

import numpy as np
import pytest

FIELDS = ("type", "rtype", "parent", "depth", "child_idx", "data")


def shuffled(tree, seed):
    """The tree's nodes in a random order: (type, rtype, parent, child_idx, data) and the
    permutation (old index -> new index)."""
    rng = np.random.default_rng(seed)
    n = tree.n
    perm = rng.permutation(n)
    par = np.where(tree.parent >= 0, perm[np.maximum(tree.parent, 0)], -1).astype(np.int32)
    out = []
    for x in (tree.type, tree.rtype, par, tree.child_idx, tree.data):
        y = np.empty_like(x)
        y[perm] = x
        out.append(y)
    return out, perm


def synth_tree(seed, fns=12, median=300.0):
    from ptilopsis_gb300.synth import SynthParams, generate
    return generate(SynthParams(seed=seed, n_functions=fns, median_fn_nodes=median))


def chain(n):
    """A path of n nodes (the deepest shape): node k's parent is k+1."""
    parent = np.arange(1, n + 1, dtype=np.int32)
    parent[-1] = -1
    child = np.zeros(n, np.int32)
    child[-1] = -1
    return (np.full(n, 3, np.uint8), np.full(n, 2, np.uint8), parent, child, np.arange(n, dtype=np.uint32))


def star(k):
    """A root with k leaf children, the root first and the leaves in reverse order."""
    n = k + 1
    parent = np.zeros(n, np.int32)
    parent[0] = -1
    child = np.zeros(n, np.int32)
    child[0] = -1
    child[1:] = np.arange(k - 1, -1, -1, dtype=np.int32)
    return (np.full(n, 7, np.uint8), np.full(n, 1, np.uint8), parent, child, np.arange(n, dtype=np.uint32) * 3)


def assert_tree(got, want, msg=""):
    for f in FIELDS:
        np.testing.assert_array_equal(getattr(got, f), getattr(want, f), err_msg=f"{msg} {f}")
    assert int(got.max_depth) == int(want.max_depth), msg


# ---------------------------------------------------------------- oracle (CPU)
def test_oracle_flatten_restores_post_order():
    from oracle import portbind
    for seed in range(4):
        t = synth_tree(0x50544E00 + seed)
        arrs, perm = shuffled(t, seed)
        ast, order = portbind.flatten(*arrs)
        assert_tree(ast, t, f"seed {seed}")
        np.testing.assert_array_equal(order[perm], np.arange(t.n))


def test_oracle_flatten_pinned_to_reference():
    from oracle import portbind, refbind
    if not refbind.available():
        pytest.skip("reference oracle not built here")
    cases = [shuffled(synth_tree(0x50544E10 + s, fns=20), s)[0] for s in range(3)] + [chain(300), star(500)]
    for k, arrs in enumerate(cases):
        assert_tree(portbind.flatten(*arrs)[0], refbind.flatten(*arrs), f"case {k}")


def _fixture_cases():
    """The reference front end's own DepthTrees (committed fixtures, built by the
    reference's DepthTree constructor), each given in a seeded random node order."""
    from conftest import ast_to_tree, load_fixture, manifest
    out = []
    for k, fx in enumerate(manifest()["fixtures"]):
        ast, _ = load_fixture(fx["name"])
        tree = ast_to_tree(ast)
        out.append((fx["name"], tree, shuffled(tree, 0x50544E60 + k)[0]))
    return out


def test_oracle_flatten_pinned_to_reference_fixtures():
    """Runs anywhere: the restatement rebuilds exactly the trees the reference built."""
    from oracle import portbind
    for name, tree, arrs in _fixture_cases():
        assert_tree(portbind.flatten(*arrs)[0], tree, name)


def test_oracle_flatten_rejects_malformed():
    from oracle import portbind
    base = list(star(5))
    for name, edit in [("two roots", lambda a: a[2].__setitem__(3, -1)),
                       ("parent out of range", lambda a: a[2].__setitem__(2, 99)),
                       ("child index taken twice", lambda a: a[3].__setitem__(2, int(a[3][1]))),
                       ("child index out of range", lambda a: a[3].__setitem__(1, 5)),
                       ("cycle", lambda a: (a[2].__setitem__(1, 2), a[2].__setitem__(2, 1)))]:
        arrs = [x.copy() for x in base]
        edit(arrs)
        with pytest.raises(portbind.PortError):
            portbind.flatten(*arrs)


# ---------------------------------------------------------------- GPU
@pytest.mark.gpu
def test_gpu_flatten_equals_oracle(built_cuda):
    from oracle import portbind
    from ptilopsis_gb300 import flatten
    cases = [shuffled(synth_tree(0x50544E20 + s, fns=4 + 9 * s), s)[0] for s in range(4)]
    cases += [chain(1), chain(5000), star(70000), shuffled(synth_tree(0x50544E30, fns=600, median=900.0), 9)[0]]
    for k, arrs in enumerate(cases):
        want, want_order = portbind.flatten(*arrs)
        got, order = flatten(*arrs)
        assert_tree(got, want, f"case {k} ({arrs[0].shape[0]} nodes)")
        np.testing.assert_array_equal(order, want_order, err_msg=f"case {k} order")


@pytest.mark.gpu
def test_gpu_flatten_reference_fixtures(built_cuda):
    from ptilopsis_gb300 import flatten
    for name, tree, arrs in _fixture_cases():
        assert_tree(flatten(*arrs)[0], tree, name)


@pytest.mark.gpu
def test_gpu_flatten_then_compile(built_cuda):
    """Flattening a shuffled tree and compiling it gives the words of the original."""
    from ptilopsis_gb300 import compile_tree, flatten
    t = synth_tree(0x50544E40, fns=40)
    arrs, _ = shuffled(t, 3)
    flat, _ = flatten(*arrs)
    np.testing.assert_array_equal(compile_tree(flat), compile_tree(t))


@pytest.mark.gpu
def test_gpu_flatten_rejects_malformed(built_cuda):
    from ptilopsis_gb300 import PtlError, flatten
    base = list(star(5))
    for name, edit in [("two roots", lambda a: a[2].__setitem__(3, -1)),
                       ("no root", lambda a: a[2].__setitem__(0, 1)),
                       ("parent out of range", lambda a: a[2].__setitem__(2, 99)),
                       ("child index taken twice", lambda a: a[3].__setitem__(2, int(a[3][1]))),
                       ("child index out of range", lambda a: a[3].__setitem__(1, 5)),
                       ("cycle", lambda a: (a[2].__setitem__(1, 2), a[2].__setitem__(2, 1)))]:
        arrs = [x.copy() for x in base]
        edit(arrs)
        with pytest.raises(PtlError) as e:
            flatten(*arrs)
        assert e.value.status == 1, name


@pytest.mark.gpu
def test_gpu_flatten_on_device_then_compile(built_cuda):
    """Device arrays in, a device DepthTree out, compiled from device memory: the words of
    the original tree, with no host copy of the flattened arrays."""
    import torch
    from ptilopsis_gb300 import RvGenerator, compile_tree, flatten
    t = synth_tree(0x50544E50, fns=30)
    arrs, perm = shuffled(t, 4)
    dev = [torch.from_numpy(x.view(np.int32) if x.dtype == np.uint32 else x).cuda() for x in arrs]
    flat, order = flatten(*dev)
    assert flat.on_device and int(flat.max_depth) == int(t.max_depth)
    assert_tree(flat.numpy(), t, "device flatten")
    np.testing.assert_array_equal(order.cpu().numpy()[perm], np.arange(t.n))
    with RvGenerator(flat) as g:
        g.process()
        np.testing.assert_array_equal(g.get_instructions(), compile_tree(t))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 7, 8, 9, 255, 4097, (1 << 20) - 1, 1 << 20])
def test_gpu_flatten_splitter_walks(built_cuda, n):
    """Random trees with and without long runs between splitters, at the sizes where the
    splitters' spacing changes: nodes in post-order, reversed and shuffled.  The tree is
    built in post-order, so the expected arrays are its own."""
    from ptilopsis_gb300 import flatten
    rng = np.random.default_rng(n)
    # a random recursive tree numbered from the root, then its post-order by one sweep
    up = np.zeros(n, np.int64)
    up[1:] = np.maximum(np.arange(1, n) - 1 - rng.integers(0, np.minimum(np.arange(1, n), 40)), 0)
    up[0] = -1
    size = np.ones(n, np.int64)
    for v in range(n - 1, 0, -1):
        size[up[v]] += size[v]
    nth, used, first = np.zeros(n, np.int64), np.zeros(n, np.int64), np.zeros(n, np.int64)
    count, depth = np.zeros(n, np.int64), np.zeros(n, np.int64)
    for v in range(1, n):  # children in number order; first: post-order index where v's subtree begins
        p = up[v]
        nth[v], count[p] = count[p], count[p] + 1
        first[v] = first[p] + used[p]
        used[p] += size[v]
        depth[v] = depth[p] + 1
    post = first + size - 1
    parent, child = np.empty(n, np.int32), np.empty(n, np.int32)
    parent[post] = np.where(up >= 0, post[np.maximum(up, 0)], -1)
    child[post] = np.where(up >= 0, nth, -1)
    type_, rtype = rng.integers(0, 40, n).astype(np.uint8), rng.integers(0, 6, n).astype(np.uint8)
    data = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    for at in (np.arange(n), np.arange(n)[::-1], rng.permutation(n)):  # node q goes to at[q]
        arrs = []
        for a in (type_, rtype, np.where(parent >= 0, at[np.maximum(parent, 0)], -1).astype(np.int32), child, data):
            b = np.empty_like(a)
            b[at] = a
            arrs.append(b)
        tree, order = flatten(*arrs)
        for name, want in (("type", type_), ("rtype", rtype), ("parent", parent), ("child_idx", child), ("data", data)):
            np.testing.assert_array_equal(getattr(tree, name), want, err_msg=name)
        want_depth = np.empty(n, np.int32)
        want_depth[post] = depth
        np.testing.assert_array_equal(tree.depth, want_depth)
        np.testing.assert_array_equal(order[at], np.arange(n))
        assert tree.max_depth == depth.max()


# ---------------------------------------------------------------- walks of any numbering
def renumbered(arrs, at):
    """The tree with node k as node at[k]."""
    out = []
    for a in (arrs[0], arrs[1], np.where(arrs[2] >= 0, at[np.maximum(arrs[2], 0)], -1).astype(np.int32), arrs[3], arrs[4]):
        b = np.empty_like(a)
        b[at] = a
        out.append(b)
    return out


def splitters_last(n):
    """A numbering of n nodes that gives the first of them the numbers that are no splitters
    (ptl_flatten.cuh's rule, enters and exits)."""
    lg = 5 if n >= 1 << 20 else 4
    top = ((np.arange(2 * n, dtype=np.uint64) * np.uint64(0x9E3779B1)) & np.uint64(0xFFFFFFFF)) >> np.uint64(32 - lg)
    splitter = (top.reshape(n, 2) == 0).any(axis=1)
    return np.concatenate([np.flatnonzero(~splitter), np.flatnonzero(splitter)])


def _walks(arrs):
    import ctypes
    from test_hostmodel import hostmodel
    parent, child = np.ascontiguousarray(arrs[2], np.int32), np.ascontiguousarray(arrs[3], np.int32)
    out = (ctypes.c_uint32 * 4)()
    hostmodel().ptlhm_flatten_walks(ctypes.c_void_p(parent.ctypes.data), ctypes.c_void_p(child.ctypes.data),
                                    ctypes.c_uint32(len(parent)), out)
    longest, most, splitters, cap = list(out)
    assert splitters <= cap
    return longest, most


def test_flatten_walks_stay_short(built):
    """A walk from one splitter to the next is bounded by the splitters' spacing, not by the
    depth or width of the tree; only numbers that follow the splitters' hash make longer
    ones (pointer jumping then ranks the tour)."""
    rng = np.random.default_rng(11)
    t = synth_tree(0x50544E70, fns=60, median=900.0)
    for arrs in (chain(1000), chain(100_000), star(100_000), (t.type, t.rtype, t.parent, t.child_idx, t.data)):
        n = len(arrs[2])
        for at in (np.arange(n), np.arange(n)[::-1], rng.permutation(n)):
            longest, most = _walks(renumbered(arrs, at))
            assert longest < most, n
    for arrs in (chain(5000), star(5000)):
        longest, most = _walks(renumbered(arrs, splitters_last(len(arrs[2]))))
        assert longest > most


@pytest.mark.gpu
@pytest.mark.parametrize("n", [700, 5000, 30_000])
def test_gpu_flatten_any_numbering(built_cuda, n):
    """Deep, wide and ordinary trees whose numbers keep the splitters to the tour's end, so
    that walks reach their limit (700 nodes: just below it), and malformed ones."""
    from oracle import portbind
    from ptilopsis_gb300 import PtlError, flatten
    t = synth_tree(0x50544E80 + n, fns=max(1, n // 900), median=900.0)
    for arrs in (chain(n), star(n - 1), (t.type, t.rtype, t.parent, t.child_idx, t.data)):
        arrs = renumbered(arrs, splitters_last(len(arrs[2])))
        want, want_order = portbind.flatten(*arrs)
        got, order = flatten(*arrs)
        assert_tree(got, want)
        np.testing.assert_array_equal(order, want_order)
    arrs = renumbered(chain(n), splitters_last(n))  # a cycle away from the root
    leaf = int(np.flatnonzero(np.bincount(arrs[2][arrs[2] >= 0], minlength=n) == 0)[0])
    above = int(arrs[2][int(arrs[2][leaf])])
    arrs[2][above] = leaf
    with pytest.raises(PtlError) as e:
        flatten(*arrs)
    assert e.value.status == 1
