"""The record form of register allocation (step records, trigger rows, lane-0 slots on one
thread, one warp, one block or a cluster) against the oracle, at the widths where the
launch changes and with symbol rings of every size.  All results are whole numbers."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from conftest import tree_to_ast
from ptilopsis_gb300.synth import SynthParams, generate


def _program(n_functions, median=40.0, seed=0x50544D00, **more):
    more = {"sigma": 1.0, "max_nesting": 6, "spill_frac": 0.25, **more}
    return generate(SynthParams(seed=seed + n_functions, n_functions=n_functions, median_fn_nodes=median, **more))


@pytest.mark.parametrize("ring", [4, 16, 1024])
@pytest.mark.parametrize("n_functions", [1, 8, 9, 40, 300])
def test_hostmodel_record_form(built, n_functions, ring):
    """The kernels' step functions on the CPU; a ring of 4 words reads most operands' symbols
    back from memory."""
    from test_hostmodel import assert_stages_equal, hostmodel
    L = hostmodel()
    L.ptlhm_set_ring_words(ctypes.c_uint32(ring))
    try:
        assert_stages_equal(tree_to_ast(_program(n_functions, 150.0, max_expr_depth=12, float_frac=0.5)))
    finally:
        L.ptlhm_set_ring_words(ctypes.c_uint32(16))


@pytest.mark.gpu
@pytest.mark.parametrize("n_functions", [1, 8, 9, 256, 257, 2048, 2049, 8192, 8193])
def test_gpu_lane0_widths(built_cuda, n_functions):
    """1 group (a lone slot), 2 and 32 (one warp), 33 and 256 (a block), 257 (a cluster of
    three CTAs), 1,024 and 1,025 (eight)."""
    from oracle import portbind
    from ptilopsis_gb300 import RvGenerator
    tree = _program(n_functions)
    ref = portbind.compile_ast(tree_to_ast(tree))
    with RvGenerator(tree) as gen:
        gen.process()
        np.testing.assert_array_equal(gen.get_instructions(), ref.words)
        t = gen.function_table()
        gen.process(row0_hash=True)  # the general form
        np.testing.assert_array_equal(gen.get_instructions(), ref.words)
        np.testing.assert_array_equal(gen.function_table()["starts"], t["starts"])


@pytest.mark.gpu
def test_gpu_batch_of_all_widths(built_cuda):
    """Programs of every width in one batch (a block per program sized by the widest, the
    widest of all on a cluster), with operands older than the batch's symbol ring."""
    from oracle import portbind
    from ptilopsis_gb300.batch import BatchCompiler
    trees = [_program(n) for n in (1, 3, 9, 257, 700, 8200)]
    trees += [_program(5, 3000.0, seed=0x50544D80 + k, max_expr_depth=12, float_frac=0.5, max_nesting=64) for k in range(3)]
    with BatchCompiler(tiles=None) as b:
        b.compile(trees)
        for k, tree in enumerate(trees):
            np.testing.assert_array_equal(b.words(k), portbind.compile_ast(tree_to_ast(tree)).words, err_msg=str(k))


@pytest.mark.parametrize("form", ["records", "records, ring of 8 words", "tiles", "serial"])
def test_hostmodel_scalar_forms(built, form):
    """The scalar generator's allocation by step records (old words read back with a small
    ring), by word tiles and in the reference's order, against its oracle."""
    from oracle import portbind
    from test_hostmodel import hostmodel
    from test_scalar import hm_compile_scalar
    L = hostmodel()
    L.ptlhm_set_ring_words(ctypes.c_uint32(8 if "8" in form else 256))
    L.ptlhm_set_scalar_tiles(1 if form == "tiles" else 0)
    try:
        for tree in (_program(9), _program(40, 150.0, max_expr_depth=12, float_frac=0.5),
                     _program(3, 2500.0, max_nesting=32, spill_frac=1.0)):
            rc, err, got = hm_compile_scalar(tree_to_ast(tree), serial=form == "serial")
            assert rc == 0, f"host model error {err}"
            np.testing.assert_array_equal(got[0], portbind.compile_ast(tree_to_ast(tree), scalar=True).words)
    finally:
        L.ptlhm_set_ring_words(ctypes.c_uint32(16))
        L.ptlhm_set_scalar_tiles(0)


@pytest.mark.gpu
@pytest.mark.parametrize("n_functions", [1, 31, 32, 33, 300])
def test_gpu_scalar_records(built_cuda, n_functions):
    """A warp's lanes partly and wholly used, functions of very different lengths side by
    side, alone and in a batch."""
    from oracle import portbind
    from ptilopsis_gb300 import RvGenerator
    from ptilopsis_gb300.batch import BatchCompiler
    tree = _program(n_functions, 300.0, max_expr_depth=12, float_frac=0.5, max_nesting=32)
    want = portbind.compile_ast(tree_to_ast(tree), scalar=True).words
    with RvGenerator(tree, scalar=True) as gen:
        gen.process()
        np.testing.assert_array_equal(gen.get_instructions(), want)
    with BatchCompiler(tiles=None, scalar=True) as b:
        b.compile([_program(5), tree, _program(2)])
        np.testing.assert_array_equal(b.words(1), want)


def _long_chain(tree, n):
    """tree with one literal operand of an addition replaced by n nested additions
    1 + (1 + (1 + ...)): n symbols that are alive at once."""
    import dataclasses
    ADD, LIT, INT = 13, 35, 2
    t, rt, par = (np.asarray(getattr(tree, k)) for k in ("type", "rtype", "parent"))
    leaf = [k for k in range(tree.n) if t[k] == LIT and rt[k] == INT and t[par[k]] == ADD][-1]
    more = 2 * n  # the leaf becomes 1, 1, .., 1 (n + 1 of them), then n additions
    at = lambda k: k if k < leaf else k + more  # the leaf's place is the outermost addition's
    cols = {k: np.asarray(getattr(tree, k)) for k in ("type", "rtype", "parent", "depth", "child_idx", "data")}
    new = {k: np.insert(c, leaf, np.zeros(more, c.dtype)) for k, c in cols.items()}
    new["parent"] = np.array([at(p) if p >= 0 else p for p in new["parent"]], cols["parent"].dtype)
    d = int(cols["depth"][leaf])
    for k in range(n + 1):  # literal k is the left operand of addition k, the last one a right one
        i = leaf + k
        new["type"][i], new["rtype"][i], new["data"][i] = LIT, INT, 1
        new["parent"][i] = leaf + more - min(k, n - 1)
        new["depth"][i], new["child_idx"][i] = d + min(k, n - 1) + 1, 1 if k == n else 0
    for k in range(n):  # addition k, the outermost last
        i = leaf + more - k
        new["type"][i], new["rtype"][i], new["data"][i] = ADD, INT, 0
        new["depth"][i] = d + k
        if k:
            new["parent"][i], new["child_idx"][i] = i + 1, 1
    return dataclasses.replace(tree, max_depth=int(new["depth"].max()), **new)


@pytest.mark.parametrize("chain", [0, 50, 70])
@pytest.mark.parametrize("n_functions", [1, 9, 130, 700])
def test_hostmodel_chunks(built, n_functions, chain):
    """The lane-0 functions in chunks; 50 nested operands fit the slots, 70 do not (the
    lock-step then does the program)."""
    from test_hostmodel import assert_stages_equal, hostmodel
    L = hostmodel()
    tree = _program(n_functions, 300.0, max_expr_depth=12, float_frac=0.3)
    locked = False
    if chain:
        tree = _program(1, 900.0, float_frac=0.0) if n_functions == 1 else tree
        tree = _long_chain(tree, chain)
    assert_stages_equal(tree_to_ast(tree))
    locked = bool(L.ptlhm_last_locked())
    if chain <= 50:
        assert not locked
    elif n_functions == 1:
        assert locked


@pytest.mark.gpu
@pytest.mark.parametrize("chain", [0, 70])
@pytest.mark.parametrize("n_functions", [1, 9, 128, 129, 1024, 1025])
def test_gpu_chunks(built_cuda, n_functions, chain):
    """Programs long enough for chunks: a lone lane-0 function, and row folds by one warp (2
    and 16 of them), four warps (17 and 128) and a block (129)."""
    from oracle import portbind
    from ptilopsis_gb300 import RvGenerator
    tree = _program(n_functions, 3000.0 if n_functions < 100 else 500.0, float_frac=0.3)
    if chain:
        tree = _long_chain(tree, chain)
    ref = portbind.compile_ast(tree_to_ast(tree))
    with RvGenerator(tree) as gen:
        gen.process()
        assert gen.function_table()["sizes"].max() > 768
        np.testing.assert_array_equal(gen.get_instructions(), ref.words)
        gen.process()  # again, in the same arrays
        np.testing.assert_array_equal(gen.get_instructions(), ref.words)


@pytest.mark.gpu
def test_gpu_batch_chunks(built_cuda):
    """A batch with programs in chunks beside short ones in lock-step, one with more symbols
    alive than there are slots, and one too wide for a block (its own launches)."""
    from oracle import portbind
    from ptilopsis_gb300.batch import BatchCompiler
    trees = [_program(n, m, float_frac=0.3) for n, m in ((1, 6000.0), (9, 4000.0), (140, 900.0), (3, 40.0), (20, 60.0))]
    trees.append(_long_chain(_program(1, 6000.0, seed=0x50544D90, float_frac=0.0), 70))
    trees.append(_program(8200, 60.0, sigma=1.5, max_fn_nodes=4000))
    with BatchCompiler(tiles=None) as b:
        for _ in range(2):
            b.compile(trees)
            for k, tree in enumerate(trees):
                np.testing.assert_array_equal(b.words(k), portbind.compile_ast(tree_to_ast(tree)).words, err_msg=str(k))
        assert max(int(b.function_table(6)["sizes"].max()), 0) > 768


@pytest.mark.parametrize("programs, threads", [(1, 512), (3, 512), (512, 512), (1000, 512), (7, 1)])
def test_hostmodel_lost_launch_fails_every_program(built, programs, threads):
    """A chunk launch that gives up a wait holds many programs: each has the error (5), so
    that none passes on words whose registers nothing allocated."""
    from test_hostmodel import hostmodel
    codes = np.zeros(programs, np.uint32)
    hostmodel().ptlhm_chunks_lost(ctypes.c_uint32(programs), ctypes.c_uint32(threads), ctypes.c_void_p(codes.ctypes.data))
    assert (codes == 5).all()


@pytest.mark.gpu
def test_gpu_chunk_wait_gives_up(built_cuda):
    """A wait of one cycle runs out: a device timeout of every program in chunks, plain and
    batched, and of no other; with the built-in wait the same objects compile again."""
    from oracle import portbind
    from ptilopsis_gb300 import PtlError, RvGenerator
    from ptilopsis_gb300.batch import BatchCompiler
    trees = [_program(n, m, float_frac=0.3) for n, m in ((9, 4000.0), (3, 40.0), (3, 6000.0), (140, 900.0))]
    refs = [portbind.compile_ast(tree_to_ast(t)).words for t in trees]
    with RvGenerator(trees[0]) as gen:
        gen.set_chunk_limits(wait_cycles=1)
        with pytest.raises(PtlError) as e:
            gen.process()
        assert e.value.status == 5
        gen.set_chunk_limits()
        gen.process()
        np.testing.assert_array_equal(gen.get_instructions(), refs[0])
    with BatchCompiler(tiles=None) as b:
        b.set_chunk_limits(wait_cycles=1)
        b.compile(trees, check=False)
        assert [b.status(k) for k in range(4)] == [5, 0, 5, 5]
        np.testing.assert_array_equal(b.words(1), refs[1])
        b.set_chunk_limits()
        b.compile(trees)
        for k, want in enumerate(refs):
            np.testing.assert_array_equal(b.words(k), want, err_msg=str(k))


@pytest.mark.parametrize("hashed", [0, 1])
@pytest.mark.parametrize("entries", [1, 64])
@pytest.mark.parametrize("n_functions", [1, 9, 130])
def test_hostmodel_general_form(built, n_functions, entries, hashed):
    """The general form, which the programs of the front end take no more: row 0 by
    definition positions where every register has one definition, and by hash, with a symbol
    cache of one entry and of many."""
    from test_hostmodel import assert_stages_equal, hostmodel
    L = hostmodel()
    L.ptlhm_set_general(1)
    L.ptlhm_set_hashed(hashed)
    L.ptlhm_set_cache_entries(ctypes.c_uint32(entries))
    try:
        assert_stages_equal(tree_to_ast(_program(n_functions, 200.0, max_expr_depth=12, float_frac=0.5)))
        assert L.ptlhm_last_hashed() == hashed
    finally:
        L.ptlhm_set_general(0)
        L.ptlhm_set_hashed(0)
        L.ptlhm_set_cache_entries(ctypes.c_uint32(4))


@pytest.mark.gpu
@pytest.mark.parametrize("n_functions", [1, 8, 9, 300, 2100])
def test_gpu_general_form(built_cuda, n_functions):
    """By definition positions (with up to 8 functions one warp does it alone) and by hash."""
    from oracle import portbind
    from ptilopsis_gb300 import RvGenerator
    tree = _program(n_functions, 200.0, max_expr_depth=12, float_frac=0.5)
    want = portbind.compile_ast(tree_to_ast(tree)).words
    with RvGenerator(tree) as gen:
        for how in ({"general": True}, {"row0_hash": True}, {"general": True}):
            gen.process(**how)
            np.testing.assert_array_equal(gen.get_instructions(), want)


# ---------------------------------------------------------------- the lane-0 lock-step
def _steps(ref):
    """Steps of the longest function, as the forms' rules count them."""
    return int(ref.bufs["cnt_fn_size"].max())


def _far_operand(tree, n):
    """tree with one literal operand of an addition replaced by 1 + (((1 + 1) + 1) + ...), n
    additions in the parentheses: the first operand is read some 3n words later (a literal is
    two words), and few symbols are alive meanwhile."""
    import dataclasses
    ADD, LIT, INT = 13, 35, 2
    t, rt, par = (np.asarray(getattr(tree, k)) for k in ("type", "rtype", "parent"))
    leaf = [k for k in range(tree.n) if t[k] == LIT and rt[k] == INT and t[par[k]] == ADD][-1]
    more = 2 * n + 2  # before the leaf, whose place is the outer addition's: 1, then 1, (1, +) n times
    at = lambda k: k if k < leaf else k + more
    cols = {k: np.asarray(getattr(tree, k)) for k in ("type", "rtype", "parent", "depth", "child_idx", "data")}
    new = {k: np.insert(c, leaf, np.zeros(more, c.dtype)) for k, c in cols.items()}
    new["parent"] = np.array([at(p) if p >= 0 else p for p in new["parent"]], cols["parent"].dtype)
    d = int(cols["depth"][leaf])

    def put(i, kind, parent, depth, child):
        new["type"][i], new["rtype"][i], new["data"][i] = kind, INT, 1 if kind == LIT else 0
        new["parent"][i], new["depth"][i], new["child_idx"][i] = parent, depth, child

    outer = leaf + more
    new["type"][outer], new["rtype"][outer], new["data"][outer] = ADD, INT, 0
    put(leaf, LIT, outer, d + 1, 0)
    add = lambda k: leaf + 3 + 2 * k  # addition k, the innermost 0
    put(leaf + 1, LIT, add(0), d + n + 1, 0)
    for k in range(n):
        depth = d + n - k
        put(add(k) - 1, LIT, add(k), depth + 1, 1)
        put(add(k), ADD, add(k + 1) if k + 1 < n else outer, depth, 0 if k + 1 < n else 1)
    return dataclasses.replace(tree, max_depth=int(new["depth"].max()), **new)


@pytest.mark.parametrize("rounds", [0, 1, 2])
@pytest.mark.parametrize("ring", [4, 16, 1024])
@pytest.mark.parametrize("n_functions", [1, 9, 40, 300])
def test_hostmodel_lock_step(built, n_functions, ring, rounds):
    """The lock-step's step functions on the CPU, several slots among them, with operands older
    than the ring: from the start, and after chunks whose rounds have run out."""
    from test_hostmodel import assert_stages_equal, hostmodel
    L = hostmodel()
    L.ptlhm_set_ring_words(ctypes.c_uint32(ring))
    L.ptlhm_set_chunks(1 if rounds else 0)
    L.ptlhm_set_chunk_rounds(ctypes.c_uint32(rounds))
    try:
        assert_stages_equal(tree_to_ast(_program(n_functions, 300.0, max_expr_depth=12, float_frac=0.5)))
        assert L.ptlhm_last_lock_step()
    finally:
        L.ptlhm_set_ring_words(ctypes.c_uint32(16))
        L.ptlhm_set_chunks(1)
        L.ptlhm_set_chunk_rounds(ctypes.c_uint32(0))


@pytest.mark.parametrize("n", [2000, 3000, 6000])
def test_hostmodel_far_operand(built, n):
    """A symbol that lives through fewer chunks than a symbol may, and through more (the
    lock-step then does the program)."""
    from test_hostmodel import assert_stages_equal, hostmodel
    tree = _far_operand(_program(1, 900.0, float_frac=0.0), n)
    assert_stages_equal(tree_to_ast(tree))
    assert bool(hostmodel().ptlhm_last_locked()) == (3 * n > 256 * 32)


@pytest.mark.gpu
@pytest.mark.parametrize("n_functions", [1, 9, 257, 2048, 2049, 4100, 8193])
def test_gpu_lock_step_short(built_cuda, n_functions):
    """Programs too short for chunks: one slot, one warp (2 slots), a block (33 and 256), a
    cluster of two CTAs (257), of three (513) and of five (1,025)."""
    from oracle import portbind
    from ptilopsis_gb300 import RvGenerator
    tree = _program(n_functions, 100.0, sigma=0.4)
    ref = portbind.compile_ast(tree_to_ast(tree), snapshots=True)
    assert _steps(ref) < 768
    with RvGenerator(tree) as gen:
        gen.process()
        np.testing.assert_array_equal(gen.get_instructions(), ref.words)


@pytest.mark.gpu
@pytest.mark.parametrize("rounds", [1, 2])
@pytest.mark.parametrize("n_functions", [1, 9, 140, 2049, 8200])
def test_gpu_lock_step_after_chunks(built_cuda, n_functions, rounds):
    """Programs long enough for chunks whose rounds have run out: operands older than the
    lock-step's ring, on one warp, a block and a cluster."""
    from oracle import portbind
    from ptilopsis_gb300 import RvGenerator
    more = {"max_expr_depth": 12, "max_nesting": 64}
    tree = _program(n_functions, 6000.0 if n_functions < 100 else 300.0, float_frac=0.3, **more)
    ref = portbind.compile_ast(tree_to_ast(tree), snapshots=True)
    assert _steps(ref) >= 768
    with RvGenerator(tree) as gen:
        gen.set_chunk_limits(rounds=rounds)
        gen.process()
        np.testing.assert_array_equal(gen.get_instructions(), ref.words)


@pytest.mark.gpu
def test_gpu_batch_lock_step_after_chunks(built_cuda):
    """A batch whose chunks' rounds run out, settled programs among them, beside one in
    lock-step from the start and one on a cluster; then with the built-in limit."""
    from oracle import portbind
    from ptilopsis_gb300.batch import BatchCompiler
    trees = [_program(n, m, float_frac=0.3) for n, m in ((1, 1500.0), (9, 4000.0), (140, 900.0), (3, 40.0))]
    trees += [_program(5, 3000.0, seed=0x50544DA0, max_expr_depth=12, float_frac=0.5, max_nesting=64)]
    trees += [_program(8200, 60.0, sigma=1.5, max_fn_nodes=4000)]
    refs = [portbind.compile_ast(tree_to_ast(t)).words for t in trees]
    with BatchCompiler(tiles=None) as b:
        for rounds in (1, 2, 0):
            b.set_chunk_limits(rounds=rounds)
            b.compile(trees)
            for k, want in enumerate(refs):
                np.testing.assert_array_equal(b.words(k), want, err_msg=f"{rounds} rounds, program {k}")


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2000, 6000])
def test_gpu_far_operand(built_cuda, n):
    """A symbol that lives through fewer chunks than a symbol may, and through more."""
    from oracle import portbind
    from ptilopsis_gb300 import RvGenerator
    tree = _far_operand(_program(9, 900.0, float_frac=0.0), n)
    ref = portbind.compile_ast(tree_to_ast(tree))
    with RvGenerator(tree) as gen:
        gen.process()
        np.testing.assert_array_equal(gen.get_instructions(), ref.words)
