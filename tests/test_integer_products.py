"""Products on the integer pipes (jit_prelude.cuh: symgbMulInt, symgbMulPow2;
codegen.cpp: mixed bodies).

On the CPU the prelude's functions themselves, compiled by g++ with the CUDA
bit intrinsics spelled out, against IEEE multiplication: equal bits for every
operand they cover, and symgbOutside true for every other.  On the GPU whole
mixed modules against the same plan below the size from which products move
(one value set), for values inside and outside the covered range."""
import ctypes as C
import re
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from symboliclib_gb300 import native

PRELUDE = ROOT / "symboliclib_gb300" / "csrc" / "engine" / "jit_prelude.cuh"
BUILD = ROOT / "symboliclib_gb300" / "_build" / "codegen_tests"

SHIM = r"""
#include <algorithm>
#include <cstdint>
#include <cstring>
using std::min;
#define __device__
#define __forceinline__ inline
static inline std::uint64_t bits(double a) { std::uint64_t u; std::memcpy(&u, &a, 8); return u; }
static inline int __double2hiint(double a) { return (int)(bits(a) >> 32); }
static inline int __double2loint(double a) { return (int)bits(a); }
static inline double __hiloint2double(int h, int l) {
    const std::uint64_t u = (std::uint64_t)(unsigned)h << 32 | (unsigned)l; double d; std::memcpy(&d, &u, 8); return d;
}
static inline unsigned __funnelshift_l(unsigned lo, unsigned hi, unsigned n) {
    n &= 31; return n ? hi << n | lo >> (32 - n) : hi;
}
"""
DRIVER = r"""
extern "C" void products(const double* a, const double* b, double* q, std::size_t n) {
    for (std::size_t i = 0; i < n; ++i) q[i] = symgbMulInt(a[i], b[i], symgbSig(a[i]), symgbSig(b[i]));
}
extern "C" void outside(const double* a, unsigned char* q, std::size_t n) {
    for (std::size_t i = 0; i < n; ++i) q[i] = symgbOutside(a[i]);
}
extern "C" void powers(const double* a, double* q, std::size_t n) {
    for (std::size_t i = 0; i < n; ++i) {
        q[4 * i] = symgbMulPow2<-1, 0>(a[i]); q[4 * i + 1] = symgbMulPow2<1, 1>(a[i]);
        q[4 * i + 2] = symgbMulPow2<-64, 1>(a[i]); q[4 * i + 3] = symgbMulPow2<64, 0>(a[i]);
    }
}
"""


@pytest.fixture(scope="module")
def lib():
    text = PRELUDE.read_text()
    parts = []
    for name in ("symgbSig", "symgbOutside", "symgbMulInt", "symgbMulPow2"):
        m = re.search(r"(?:template <[^>]*>\n)?__device__ __forceinline__ \w+ " + name + r"\(.*?\n}\n", text, re.S)
        parts.append(m.group(0))
    BUILD.mkdir(parents=True, exist_ok=True)
    src, out = BUILD / "products.cpp", BUILD / "products.so"
    src.write_text(SHIM + "".join(parts) + DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", str(src), "-o", str(out)],
                   check=True, capture_output=True)
    return C.CDLL(str(out))


def product(lib, a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    q = np.empty_like(a)
    lib.products(a.ctypes.data_as(C.c_void_p), b.ctypes.data_as(C.c_void_p), q.ctypes.data_as(C.c_void_p),
                 C.c_size_t(a.size))
    return q


def values(rng, n, lo=-255, hi=256, bits=52):
    """+-[2^lo, 2^hi), significands with `bits` random bits below the leading one."""
    m = (rng.integers(0, 1 << 52, n, dtype=np.uint64) >> np.uint64(52 - bits)) << np.uint64(52 - bits)
    e = rng.integers(1023 + lo, 1023 + hi, n).astype(np.uint64)
    return (rng.integers(0, 2, n, dtype=np.uint64) << np.uint64(63) | e << np.uint64(52) | m).view(np.float64)


def same(a, b):
    return np.array_equal(a.view(np.uint64), b.view(np.uint64))


EDGES = np.array([1.0, np.nextafter(1, 2), np.nextafter(2, 1), 1.5, 3.0, 2.0 ** -255, np.nextafter(2.0 ** 256, 0), 0.0,
                  np.sqrt(2.0), np.nextafter(np.sqrt(2.0), 2), 1 + 2.0 ** -26, 1 + 2.0 ** -27, 2 - 2.0 ** -25])


@pytest.mark.parametrize("abits,bbits", [(52, 52), (26, 26), (27, 26), (20, 32), (21, 32), (1, 52), (0, 0), (32, 21)])
def test_products_equal_ieee(lib, abits, bbits):
    """Short significands make exact ties and exact products frequent."""
    rng = np.random.default_rng(abits * 64 + bbits)
    a, b = values(rng, 400000, bits=abits), values(rng, 400000, bits=bbits)
    assert same(product(lib, a, b), a * b)


def test_products_of_edges_zeros_and_up_to_four_factors(lib):
    e = np.concatenate([EDGES, -EDGES])
    a, b = (x.ravel() for x in np.meshgrid(e, e))
    ab = a * b
    assert same(product(lib, a, b), ab)
    inside = np.concatenate([EDGES, -EDGES, values(np.random.default_rng(1), 500)])
    rng = np.random.default_rng(2)
    f = [rng.choice(inside, 300000) for _ in range(4)]
    with np.errstate(under="raise", over="raise"):
        two, other = f[0] * f[1], f[2] * f[3]
        three, four = two * f[2], two * other
        chain = three * f[3]
    assert same(product(lib, two, f[2]), three)
    assert same(product(lib, two, other), four)
    assert same(product(lib, three, f[3]), chain)


def test_outside_covers_everything_else(lib):
    rng = np.random.default_rng(3)
    any_bits = rng.integers(0, 1 << 64, 400000, dtype=np.uint64).view(np.float64)
    special = np.array([np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.0 ** -1022, 2.0 ** 256, np.nextafter(2.0 ** -255, 0),
                        1e-310, -2.0 ** 300])
    a = np.concatenate([any_bits, special, EDGES, -EDGES, values(rng, 1000)])
    q = np.empty(a.size, np.uint8)
    lib.outside(a.ctypes.data_as(C.c_void_p), q.ctypes.data_as(C.c_void_p), C.c_size_t(a.size))
    covered = (a == 0) | ((np.abs(a) >= 2.0 ** -255) & (np.abs(a) < 2.0 ** 256))
    assert np.array_equal(q.astype(bool), ~covered)


def test_powers_of_two(lib):
    a = np.concatenate([EDGES, -EDGES, values(np.random.default_rng(4), 100000)])
    q = np.empty((a.size, 4))
    lib.powers(a.ctypes.data_as(C.c_void_p), q.ctypes.data_as(C.c_void_p), C.c_size_t(a.size))
    assert same(np.ascontiguousarray(q.T), np.stack([a * 0.5, a * -2.0, a * -2.0 ** -64, a * 2.0 ** 64]))


PLAIN, LEVELS, PERSISTENT = native.SCHEDULE_PLAIN, native.SCHEDULE_LEVELS, native.SCHEDULE_PERSISTENT


@pytest.mark.gpu
@pytest.mark.parametrize("name,size,sets,math,kind", [
    ("cotan", 14, 56, native.MATH_FAST, PLAIN), ("cotan", 14, 56, native.MATH_FAST, PERSISTENT),
    ("cotan", 14, 56, native.MATH_EXACT, LEVELS), ("cloth", 10, 112, native.MATH_FAST, LEVELS),
    ("cloth", 10, 112, native.MATH_EXACT, PLAIN), ("cloth", 10, 112, native.MATH_FAST, PERSISTENT),
    ("neohookean", 2, 432, native.MATH_FAST, LEVELS)])
def test_mixed_modules_equal_fp64_modules(name, size, sets, math, kind):
    """Every value set of a module with integer products gives the bits of its
    own one-set run (too few work items for them), also where values leave the
    covered range (another scale, zeros, infinities, NaN, subnormals)."""
    w = native.Workload(name, size, 6)
    rng = np.random.default_rng(size)
    scale = [1.0, 1e-90, 1e100, 0.0, np.inf, np.nan, 1e-310, -1.0]
    kinds = len(scale)
    per = [[a * (scale[s] if s < kinds else 1.0) * (1 + 1e-3 * rng.uniform(-1, 1, a.size)) for s in range(2 * kinds)]
           for a in w.inputs]
    for a in per:  # single entries out of range in otherwise ordinary sets
        for s in range(kinds, 2 * kinds):
            a[s][rng.integers(0, a[s].size, 3)] = scale[s - kinds]
    u = native.Unit.from_workload(w)
    u.set_num_sets(sets)
    u.set_schedule(kind=kind, math=math)
    src = u.compiled_source(kind)
    assert "symgbMulInt(v" in src
    for i, a in enumerate(per):
        u.set_arg(i, np.stack([a[s % (2 * kinds)] for s in range(sets)]).ravel())
    u.run()
    out = u.get_result(0).reshape(sets, -1)
    one = native.Unit.from_workload(w)
    one.set_schedule(kind=kind, math=math)
    assert "symgbMulInt(v" not in one.compiled_source(kind)
    for s in range(2 * kinds):
        for i, a in enumerate(per):
            one.set_arg(i, a[s])
        one.run()
        ref = one.get_result(0)
        for t in range(s, sets, 2 * kinds):
            assert np.array_equal(out[t].view(np.uint64), ref.view(np.uint64)), (s, t)
