"""Forms of the compiled executor's bodies that other tests do not reach: mixed
bodies with several work items per thread (a heavy one's loop is rolled), for
values inside and outside what the integer products cover; templates in pieces
with and without direct result rows, in both math modes."""
import re

import numpy as np
import pytest

from symboliclib_gb300 import native

pytestmark = pytest.mark.gpu

PLAIN, LEVELS, PERSISTENT = native.SCHEDULE_PLAIN, native.SCHEDULE_LEVELS, native.SCHEDULE_PERSISTENT


@pytest.mark.parametrize("name,size,sets,math,kind,items,rolled", [
    ("cloth", 10, 112, native.MATH_FAST, PLAIN, 4, True), ("cloth", 10, 112, native.MATH_EXACT, LEVELS, 2, True),
    ("cotan", 14, 56, native.MATH_FAST, LEVELS, 2, False)])
def test_mixed_bodies_with_several_items_per_thread(name, size, sets, math, kind, items, rolled):
    """Ordinary value sets and, among them, sets with zeros, infinities, NaN,
    subnormals or another scale, whole or in single entries: the bits of a
    module of one set, which has no integer products."""
    w = native.Workload(name, size, 6)
    rng = np.random.default_rng(size)
    scale = [1.0, 1e-90, 0.0, np.inf, np.nan, 1e-310]
    kinds = len(scale)
    per = [[a * (scale[s] if s < kinds else 1.0) * (1 + 1e-3 * rng.uniform(-1, 1, a.size)) for s in range(2 * kinds)]
           for a in w.inputs]
    for a in per:
        for s in range(kinds, 2 * kinds):
            a[s][rng.integers(0, a[s].size, 3)] = scale[s - kinds]
    u = native.Unit.from_workload(w)
    u.set_num_sets(sets)
    u.set_schedule(kind=kind, math=math, items_per_thread=items, threads_per_block=64)
    src = u.compiled_source(kind)
    assert "symgbMulInt(v" in src and ("#pragma unroll 1\n" in src) == rolled
    for i, a in enumerate(per):
        u.set_arg(i, np.stack([a[s % (2 * kinds)] for s in range(sets)]).ravel())
    u.run()
    out = u.get_result(0).reshape(sets, -1)
    one = native.Unit.from_workload(w)
    one.set_schedule(kind=kind, math=math, items_per_thread=items, threads_per_block=64)
    assert "symgbMulInt(v" not in one.compiled_source(kind)
    for s in range(2 * kinds):
        for i, a in enumerate(per):
            one.set_arg(i, a[s])
        one.run()
        ref = one.get_result(0)
        for t in range(s, sets, 2 * kinds):
            assert np.array_equal(out[t].view(np.uint64), ref.view(np.uint64)), (s, t)


@pytest.mark.parametrize("math", [native.MATH_FAST, native.MATH_EXACT])
@pytest.mark.parametrize("name,size,kind", [("cloth", 6, PLAIN), ("cloth", 6, PERSISTENT), ("neohookean", 2, LEVELS)])
def test_pieces_equal_the_interpreter(name, size, kind, math):
    w = native.Workload(name, size, 6)
    u = native.Unit.from_workload(w)
    u.set_schedule(kind=kind, math=math, executor=native.EXEC_INTERPRETER)
    for i, a in enumerate(w.inputs):
        u.set_arg(i, a)
    u.run()
    ref = u.get_result(0)
    u.set_schedule(kind=kind, math=math)
    for direct in (False, True):
        u.set_direct_outputs(direct)
        src = u.compiled_source(kind)
        assert "symgbPart" in src and ("res[" in src) == direct
        u.run()
        assert np.array_equal(u.get_result(0).view(np.uint64), ref.view(np.uint64)), direct


def make_in_place(w, k, access):
    """The workload's plan with access `access` of kernel k naming the slot of
    the instance's own first output row, which is so read and then overwritten
    in every run.  Returns the index table."""
    d = w.plan.contents
    kd = d.kernels[k]
    n, rows = int(kd.num_instances), int(kd.num_index_rows)
    at = int(kd.index_offset)
    table = np.concatenate([w.index_data, w.index_data[at:at + n * rows],
                            np.arange(kd.output_offset, kd.output_offset + n, dtype=np.uint32)]).astype(np.uint32)
    kd.index_offset, kd.num_index_rows = len(w.index_data), rows + 1
    kd.access[2 * access], kd.access[2 * access + 1] = rows, 0
    d.num_indices = len(table)
    return table


@pytest.mark.parametrize("name,size,k,sets,form", [("neohookean", 2, 0, 1, "symgbPart"), ("cloth", 6, 1, 1, "symgbPart"),
                                                   ("cloth", 10, 1, 112, "symgbMixed")])
def test_kernels_that_overwrite_what_they_read(name, size, k, sets, form):
    """Such a kernel keeps one body: another piece, or an item evaluated again,
    would read what has been stored."""
    w = native.Workload(name, size, 6)
    whole = native.Unit.from_workload(w, init=False)
    whole.set_num_sets(sets)
    assert re.search(rf"{form}{k}(?!\d)", whole.compiled_source(PLAIN))
    table = make_in_place(w, k, 2)
    units = []
    for executor in (native.EXEC_COMPILED, native.EXEC_INTERPRETER):
        u = native.Unit(w.plan, table, w.out_index_data, w.const_data)
        u.set_num_sets(sets)
        u.set_schedule(kind=PLAIN, math=native.MATH_EXACT, executor=executor)
        units.append(u)
    assert not re.search(rf"{form}{k}(?!\d)", units[0].compiled_source(PLAIN))
    rng = np.random.default_rng(size)
    for _ in range(4):
        results = []
        ins = [np.stack([a * (1e-90 if s % 5 == 3 else 1.0) * (1 + 1e-3 * rng.uniform(-1, 1, a.size))
                         for s in range(sets)]).ravel() for a in w.inputs]
        for u in units:
            for i, a in enumerate(ins):
                u.set_arg(i, a)
            u.run()
            results.append(u.get_result(0))
        a, b = results
        assert np.array_equal(np.isnan(a), np.isnan(b)) and np.isfinite(a).any()
        ok = ~np.isnan(a)
        assert np.array_equal(a[ok].view(np.uint64), b[ok].view(np.uint64))
