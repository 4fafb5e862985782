"""Templates cut into pieces (codegen.cpp: templatePieces): every kernel's
pieces, compiled for the host as in test_codegen_cpu.py and run one after
another over every work item, store exactly the results of the whole body."""
import ctypes as C
import hashlib
import re
import subprocess

import numpy as np
import pytest

from symboliclib_gb300 import native
from test_codegen_cpu import BUILD, HOST_SHIM

import oracle.cpu as ocpu

SHIM = HOST_SHIM + """
#define SYMGB_ORDERED
template <int O> static inline const double* symgbOrder(const double* x) { return x; }
"""


def run_pieces(w, inputs, kind, math, sets, tpb):
    u = native.Unit.from_workload(w, init=False)
    u.set_num_sets(sets)
    u.set_schedule(kind=kind, math=math, threads_per_block=tpb)
    src = u.compiled_source(kind)
    bodies = src[src.index("// kernel 0:"):src.index('extern "C"')]
    d = w.plan.contents
    calls, cut = [], 0
    for k in range(d.num_kernels):
        parts = sorted({int(q) for q in re.findall(rf"symgbPart{k}_(\d+)\(", bodies)})
        cut += len(parts) > 1
        names = [f"symgbPart{k}_{q}" for q in parts] or [f"symgbBody{k}"]
        if f"symgbBody{k}(" in bodies:
            run = " ".join(f"{f}<0>(x, xw, p, c, nullptr, nullptr, i, s);" for f in names)
            calls.append(f"case {k}: {run} break;")
    text = SHIM + bodies + ('extern "C" void run(int k, const double* x, double* xw, const unsigned* p, const double* c, '
                            "unsigned long long n, unsigned S) { for (unsigned long long i = 0; i < n; ++i) "
                            "for (unsigned s = 0; s < S; ++s) switch (k) {" + " ".join(calls) + "} }\n")
    BUILD.mkdir(parents=True, exist_ok=True)
    tag = hashlib.sha1(text.encode()).hexdigest()[:16]
    path, lib = BUILD / f"pieces_{tag}.cpp", BUILD / f"pieces_{tag}.so"
    if not lib.exists():
        path.write_text(text)
        subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-fno-fast-math", "-shared", "-fPIC",
                        str(path), "-o", str(lib)], check=True, capture_output=True)
    h = C.CDLL(str(lib))
    x = np.full(int(d.num_total_memory) * sets, np.nan)
    for i, a in enumerate(inputs):
        at = int(d.arg_start[i])
        for s in range(sets):
            x[(at + np.arange(a.shape[1])) * sets + s] = a[s]
    p = np.ascontiguousarray(w.index_data if len(w.index_data) else np.zeros(1), np.uint32)
    c = np.ascontiguousarray(w.const_data if len(w.const_data) else np.zeros(1), np.float64)
    for k in range(d.num_kernels):
        h.run(k, *(C.c_void_p(v.ctypes.data) for v in (x, x, p, c)), C.c_ulonglong(int(d.kernels[k].num_instances)),
              C.c_uint(sets))
    ids = w.out_index_data.astype(np.int64)
    return np.stack([x[ids * sets + s] for s in range(sets)]), cut


@pytest.mark.parametrize("kind", [native.SCHEDULE_PLAIN, native.SCHEDULE_LEVELS, native.SCHEDULE_PERSISTENT])
@pytest.mark.parametrize("name,size,sets,tpb", [("cloth", 3, 1, 128), ("cloth", 8, 3, 64), ("cloth", 12, 4, 128),
                                                ("neohookean", 1, 1, 128), ("neohookean", 3, 2, 256)])
def test_pieces_store_the_whole_templates_results(name, size, sets, tpb, kind):
    w = native.Workload(name, size, 8)
    rng = np.random.default_rng(size)
    inputs = [np.stack([a * (1 + 1e-3 * rng.uniform(-1, 1, a.size)) for _ in range(sets)]) for a in w.inputs]
    out, cut = run_pieces(w, inputs, kind, native.MATH_EXACT, sets, tpb)
    assert cut  # these leave schedulers idle
    for s in range(sets):
        ref = ocpu.evaluate(w.plan, w.index_data, w.out_index_data, w.const_data, [a[s] for a in inputs])[0]
        assert np.array_equal(out[s].view(np.uint64), ref.view(np.uint64)), s


def test_full_chips_and_light_templates_stay_whole():
    for name, size, sets in (("cloth", 40, 64), ("cotan", 40, 1), ("ata", 30, 1)):
        u = native.Unit.from_workload(native.Workload(name, size, 8), init=False)
        u.set_num_sets(sets)
        for kind in range(3):
            assert "symgbPart" not in u.compiled_source(kind)
