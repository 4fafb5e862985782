"""Order of the compiled executor's launches.

A launch reads what earlier launches wrote.  Its own griddepcontrol.wait is
what makes those writes visible to it, so every generated kernel waits before
its first read of x, whatever the dependency levels of its neighbours.  Launches
that a replayed plain run puts side by side are chosen from what the tables make
them read and write, not from the plan's level numbers."""
import functools
import re
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from symboliclib_gb300 import build, native

import oracle.cpu as ocpu

PLAIN, LEVELS, PERSISTENT = native.SCHEDULE_PLAIN, native.SCHEDULE_LEVELS, native.SCHEDULE_PERSISTENT


@functools.lru_cache(None)
def workload(name, size):
    return native.Workload(name, size, 8)


def entries(src):
    """Name and body text of every kernel of a generated module."""
    for m in re.finditer(r'extern "C" __global__ void __launch_bounds__\([^)]*\) (\w+)\(.*?\n}\n', src, re.S):
        yield m.group(1), m.group(0)[m.group(0).index("{"):]


@pytest.mark.parametrize("kind", [PLAIN, LEVELS, PERSISTENT])
@pytest.mark.parametrize("items,layout", [(1, native.ITEMS_STRIDED), (4, native.ITEMS_STRIDED), (2, native.ITEMS_GROUPED)])
@pytest.mark.parametrize("name,size,sets", [("cloth", 8, 1), ("cloth", 20, 64), ("ata", 9, 1), ("cotan", 8, 1),
                                            ("neohookean", 2, 3)])
def test_every_launch_waits_before_it_reads(name, size, sets, items, layout, kind):
    u = native.Unit.from_workload(workload(name, size), init=False)
    u.set_num_sets(sets)
    native.check(u._lib.symgb_set_item_layout(u.handle, layout))
    u.set_schedule(kind=kind, items_per_thread=items)
    src = u.compiled_source(kind)
    waits = re.search(r"template <int ORDER>.*?symgbOrder.*?\n}", src, re.S).group(0)
    assert re.search(r"if \(ORDER(?: & 1)?\) asm volatile\(\"griddepcontrol.wait;\" : \"\+l\"\(x\)", waits)
    found = 0
    for kernel, body in entries(src):
        calls = list(re.finditer(r"symgb(?:Body|Mixed|Part|Group)\d+(?:_\d+)?<([^>]*)>\(", body))
        assert calls, kernel
        first = body[:calls[0].start()]
        before = "x = symgbOrder<1>(x);" in first or "symgbDependencyWait();" in first
        for c in calls:
            inside = "Group" not in c.group(0) and int((c.group(1) + ", 0").split(",")[1]) & 1
            assert before or inside, (kernel, c.group(0))
        found += 1
    assert found


def test_copy_kernels_read_what_may_change_with_ordinary_loads():
    """Kernels that start before their predecessor has ended do not read its
    results through the read-only path."""
    found = 0
    for path in (build.CSRC / "engine").glob("*.cu*"):
        for m in re.finditer(r"__global__ [^;{]*?\((.*?)\) \{(.*?)\n}", path.read_text(), re.S):
            for p in re.findall(r"symgbOrder<1>\((\w+)\)", m.group(2)):
                found += 1
                assert not re.search(rf"__ld\w+\({p}\b", m.group(2)), (path.name, p)
                assert not re.search(rf"__restrict__ {p}\b", m.group(1)), (path.name, p)
    assert found >= 5


@pytest.mark.parametrize("kind", [PLAIN, LEVELS, PERSISTENT])
@pytest.mark.parametrize("path", [native.LOAD_READONLY, native.LOAD_L1, native.LOAD_L2])
def test_generated_kernels_read_x_with_ordinary_loads(path, kind):
    """x is written while a chained launch is already resident, so no load path
    reads it through the read-only path."""
    u = native.Unit.from_workload(workload("cloth", 8), init=False)
    u.set_load_path(path)
    src = u.compiled_source(kind)
    load = re.search(r"double symgbLoadX\(const double\* a\) \{\n(.*?)\n}", src, re.S).group(1)
    assert load.strip() == f"return L2 ? __ldcg(a) : {'__ldcg' if path == native.LOAD_L2 else '__ldca'}(a);"
    assert not re.search(r"(SYMGB_LD|__ldg)\(x\b", src)


def test_side_by_side_kernels_share_no_written_slot():
    out, lib = build.OBJ / "beside_earlier_test", build.LIB
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'include'}", f"-I{build.CSRC / 'engine'}",
                    str(ROOT / "tests" / "cpp" / "beside_earlier.cpp"), "-o", str(out), f"-L{lib}", "-lsymgb",
                    f"-Wl,-rpath,{lib}"], check=True, capture_output=True, text=True)
    r = subprocess.run([str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("careless", [False, True])
@pytest.mark.parametrize("name,size", [("cotan", 8), ("cloth", 12), ("ata", 9), ("neohookean", 2)])
def test_plain_runs_need_no_levels(name, size, careless):
    """Plain runs evaluate the kernels in plan order, also when every kernel
    claims the same level: the first run launch by launch, the others replayed."""
    w = native.Workload(name, size, 5)
    rng = np.random.default_rng(size)
    runs = []
    for _ in range(4):
        ins = [a * (1 + 1e-3 * rng.uniform(-1, 1, a.size)) for a in w.inputs]
        runs.append((ins, ocpu.evaluate(w.plan, w.index_data, w.out_index_data, w.const_data, ins)[0]))
    if careless:
        for k in range(w.plan.contents.num_kernels):
            w.plan.contents.kernels[k].level = 0
    u = native.Unit.from_workload(w)
    u.set_schedule(kind=PLAIN, math=native.MATH_EXACT)
    for ins, ref in runs:
        for i, a in enumerate(ins):
            u.set_arg(i, a)
        u.run()
        assert np.array_equal(u.get_result(0).view(np.uint64), ref.view(np.uint64))
