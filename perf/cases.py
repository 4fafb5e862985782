"""Performance cases of the engine: what a program does with it, through the
public entry points, over the range of sizes, value sets, data paths and
options it is used with.

A case is a dict of plain values; its "what" names the path:

  assemble   inputs of a planned unit set, evaluated, results read
  batch      many units of uneven size replayed as one CUDA graph
  solve      batched Krylov solve with the assembled matrix's pattern
  train      epochs of the schedule cost model

Plans are built by the front end once per process and kept, as a program that
evaluates one sparsity pattern many times keeps them, together with the unit
made from them; the values (vertex positions, velocities, matrix entries,
right-hand sides, training samples) are made anew from the seed of every
prepare() and are other values in every value set.
"""
from __future__ import annotations

import ctypes as C
import json
import math

import numpy as np
import torch

from symboliclib_gb300 import native

SCHEDULES = {"plain": native.SCHEDULE_PLAIN, "levels": native.SCHEDULE_LEVELS,
             "persistent": native.SCHEDULE_PERSISTENT}
PLAN_SEED = 2024


def _assemble(name, plan, size, sets=1, math="fast", schedule="levels", tpb=128, items=1, io="device",
              executor="compiled"):
    return {"name": name, "what": "assemble", "plan": plan, "size": size, "sets": sets, "math": math,
            "schedule": schedule, "tpb": tpb, "items": items, "io": io, "executor": executor}


def listed():
    return [
        # A small mesh edited interactively: one Laplacian per call with host
        # arrays, default schedule.  Latency, launches and transfers.
        _assemble("cotan_16_host", "cotan", 16, schedule="plain", io="host"),
        # The Laplacian of an ordinary mesh that stays on the device.
        _assemble("cotan_100", "cotan", 100, tpb=256),
        # A large mesh (714 k nonzeros), the single-set device benchmark's shape and schedule.
        _assemble("cotan_320", "cotan", 320, tpb=256),
        # One implicit cloth step: one state per call, one launch per kernel.
        _assemble("cloth_64", "cloth", 64, schedule="plain"),
        # The batched headline workload's family, 64 states at once, in the
        # schedule its tuning chooses.  The largest.
        _assemble("cloth_100_x64", "cloth", 100, sets=64, schedule="plain", tpb=64, items=4),
        # Results that must equal the reference's bit for bit: exact mode, a few states.
        _assemble("cloth_41_x8_exact", "cloth", 41, sets=8, math="exact"),
        # Hessian of a tetrahedral solid from differentiated energies: a few large templates.
        _assemble("neohookean_8_x4", "neohookean", 8, sets=4),
        # Sparse matrix algebra at the size of the reference's CPU example, host arrays, exact.
        _assemble("ata_100_host_exact", "ata", 100, math="exact", schedule="plain", io="host"),
        # No run-time compiler wanted: the precompiled interpreter.
        _assemble("cloth_31_x4_interpreter", "cloth", 31, sets=4, executor="interpreter"),
        # A scene of eight garments of uneven size and state count, one graph replay.
        {"name": "cloth_batch_8", "what": "batch", "count": 8, "smallest": 8, "largest": 45, "most_sets": 16,
         "math": "fast", "streams": 8},
        # Implicit step's linear solve, eight states, vertex-block preconditioner.
        {"name": "solve_bicgstab_100_x8", "what": "solve", "side": 100, "sets": 8, "method": "bicgstab", "block": 3},
        # Fitting the schedule cost model to the timings of some twenty units.
        {"name": "train_2500", "what": "train", "samples": 2500, "features": 50, "hidden": 64, "epochs": 4},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["assemble"] * 6 + ["solve", "solve", "train", "batch"])
    if kind == "solve":
        method = rng.choice(["cg", "bicgstab"])
        side = _log_int(rng, 8, 100)
        return {"what": "solve", "side": side, "sets": _log_int(rng, 1, 8), "method": method,
                "block": rng.choice([1, 3]) if method == "bicgstab" else 1}
    if kind == "train":
        return {"what": "train", "samples": _log_int(rng, 100, 2500), "features": rng.randint(20, 50),
                "hidden": rng.choice([32, 48, 64]), "epochs": rng.randint(1, 4)}
    if kind == "batch":
        return {"what": "batch", "count": rng.randint(2, 8), "smallest": rng.randint(5, 10),
                "largest": rng.randint(20, 45), "most_sets": rng.randint(1, 16),
                "math": rng.choice(["fast", "fast", "exact"]), "streams": rng.choice([2, 4, 8])}
    plan = rng.choice(["cotan", "cotan", "cloth", "cloth", "cloth", "neohookean", "ata"])
    lo, hi, most = {"cotan": (12, 320, 64), "cloth": (6, 100, 64), "neohookean": (2, 8, 16), "ata": (10, 200, 16)}[plan]
    size = _log_int(rng, lo, hi)
    # no more work than the largest listed case of the family
    room = {"cotan": 320 ** 2 * 8, "cloth": 100 ** 2 * 64, "neohookean": 8 ** 3 * 16, "ata": 200 ** 2 * 8}[plan]
    power = 3 if plan == "neohookean" else 2
    sets = 1 if rng.random() < 0.4 else _log_int(rng, 1, max(1, min(most, room // size ** power)))
    schedule = rng.choice(["plain", "levels", "levels", "persistent"]) if plan != "neohookean" else "plain"
    case = _assemble("", plan, size, sets, rng.choice(["fast", "fast", "fast", "exact"]), schedule,
                     rng.choice([64, 128, 256]), rng.choice([1, 1, 2, 4]), rng.choice(["device", "device", "host"]),
                     rng.choice(["compiled"] * 5 + ["interpreter"]))
    del case["name"]
    return case


# ---------------------------------------------------------------- what a program keeps

_kept: dict = {}


def _keep(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _plan(name, size):
    return _keep(("plan", name, size), lambda: native.Workload(name, size, PLAN_SEED))


def _stream():
    return _keep("stream", torch.cuda.Stream)


def _unit(plan, size, sets, schedule, math, tpb, items, executor):
    u = native.Unit.from_workload(_plan(plan, size))
    native.check(u._lib.symgb_set_stream(u.handle, C.c_void_p(_stream().cuda_stream)))
    if sets > 1:
        u.set_num_sets(sets)
    u.set_schedule(kind=SCHEDULES[schedule], math=native.MATH_FAST if math == "fast" else native.MATH_EXACT,
                   threads_per_block=tpb, items_per_thread=items,
                   executor=native.EXEC_COMPILED if executor == "compiled" else native.EXEC_INTERPRETER)
    u.prepare()
    return u


# ---------------------------------------------------------------- values

def _values(plan, size, sets, rng):
    """Input containers [sets, length] of a plan: the workload's state moved a
    little, another way in every set."""
    base = _plan(plan, size).inputs
    if plan == "cotan":  # vertex positions of a jittered unit-square grid
        return [base[0] + rng.uniform(-0.05, 0.05, (sets, base[0].size)) / size]
    if plan == "cloth":  # positions at unit spacing, velocities
        return [base[0] + rng.uniform(-0.02, 0.02, (sets, base[0].size)),
                rng.uniform(-0.1, 0.1, (sets, base[1].size))]
    if plan == "neohookean":  # positions at unit spacing
        return [base[0] + rng.uniform(-0.01, 0.01, (sets, base[0].size))]
    return [rng.uniform(-1.0, 1.0, (sets, a.size)) for a in base]  # matrix entries


def _batch_members(case):
    """(side, sets) of every unit: log-uniform sides, 1 .. most_sets states."""
    n = case["count"]
    ratio = case["largest"] / case["smallest"]
    return [(round(case["smallest"] * ratio ** (k / max(1, n - 1))), 1 + (5 * k) % case["most_sets"]) for k in range(n)]


def _cloth_pattern(side):
    """Lower-triangle CSC pattern of a cloth matrix: every vertex couples to
    itself, its edge neighbours and the vertices opposite its edges, in all
    three coordinates (stored n apart)."""
    n = side * side
    j, i = np.divmod(np.arange(n), side)
    pairs = []
    for dx, dy in [(0, 0), (1, 0), (0, 1), (1, 1), (1, -1), (2, 1), (1, 2)]:
        for sx in ((1, -1) if (dx, dy) != (0, 0) else (1,)):
            a, b = i + sx * dx, j + sx * dy
            ok = (a >= 0) & (a < side) & (b >= 0) & (b < side)
            pairs.append(np.stack([np.arange(n)[ok], (a + b * side)[ok]]))
    r, c = np.concatenate(pairs, 1)
    rows = np.concatenate([r + p * n for p in range(3) for _ in range(3)])
    cols = np.concatenate([c + q * n for _ in range(3) for q in range(3)])
    low = rows >= cols
    rows, cols = rows[low], cols[low]
    order = np.lexsort((rows, cols))
    rows, cols = rows[order], cols[order]
    cp = np.zeros(3 * n + 1, np.int64)
    np.add.at(cp, cols + 1, 1)
    return 3 * n, np.cumsum(cp), rows.astype(np.int32), cols.astype(np.int32)


def _system(case, rng):
    """Values [sets, nnz] of symmetric positive definite systems (mass and
    stiffness of an implicit step: dominant diagonals of uneven size) and
    right-hand sides [sets, n]."""
    n, cp, ri, ci = _keep(("pattern", case["side"]), lambda: _cloth_pattern(case["side"]))
    S = case["sets"]
    off = ri != ci
    v = rng.uniform(-1.0, 0.2, (S, ri.size))
    diag = np.zeros((S, n))
    for s in range(S):
        w = np.abs(v[s, off])
        diag[s] = np.bincount(ri[off], w, n) + np.bincount(ci[off], w, n)
    v[:, ~off] = (diag * rng.uniform(1.02, 1.3, (S, n)))[:, ci[~off]]
    return v, rng.standard_normal((S, n))


def _samples(case, rng):
    """Standardised features, log times and starting weights of the cost model."""
    n, f, h = case["samples"], case["features"], case["hidden"]
    X = rng.standard_normal((n, f)).astype(np.float32)
    y = (3.0 + X[:, 0] * X[:, 1] + np.sin(2.0 * X[:, 2]) + 0.1 * rng.standard_normal(n)).astype(np.float32)
    a, b = math.sqrt(6.0 / f), math.sqrt(6.0 / h)
    p = np.concatenate([rng.uniform(-a, a, f * h), np.zeros(h), rng.uniform(-b, b, h * h), np.zeros(h),
                        rng.uniform(-b, b, h), np.zeros(1)]).astype(np.float32)
    return X, y, p


def _key(case):
    return json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)


def _device(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# ---------------------------------------------------------------- cases

LEARNING_RATE = 3e-3
TOLERANCE = 1e-11


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    s = {"what": case["what"], "case": case}
    if case["what"] == "assemble":
        u = _keep(_key(case), lambda: _unit(case["plan"], case["size"], case["sets"], case["schedule"], case["math"],
                                            case["tpb"], case["items"], case["executor"]))
        s["unit"] = u
        ins = _values(case["plan"], case["size"], case["sets"], rng)
        if case["io"] == "host":
            s["inputs"] = ins
        else:
            s["inputs"] = [_device(a) for a in ins]
            s["out"] = torch.empty((case["sets"], u.output_length[0]), dtype=torch.float64, device="cuda")
    elif case["what"] == "batch":
        def make():
            units = [_unit("cloth", side, sets, "levels", case["math"], 128, 1, "compiled")
                     for side, sets in _batch_members(case)]
            handles = (C.c_void_p * len(units))(*[u.handle.value for u in units])
            b = C.c_void_p()
            native.check(native.symgb().symgb_batch_create(handles, len(units), case["streams"], C.byref(b)))
            return units, b
        s["units"], s["batch"] = _keep(_key(case), make)
        s["inputs"] = [[_device(a) for a in _values("cloth", side, sets, rng)] for side, sets in _batch_members(case)]
        s["out"] = [torch.empty((sets, u.output_length[0]), dtype=torch.float64, device="cuda")
                    for u, (_, sets) in zip(s["units"], _batch_members(case))]
    elif case["what"] == "solve":
        v, b = _system(case, rng)

        def make():
            n, cp, ri, _ = _kept[("pattern", case["side"])]
            solver = native.SparseSolver(n, cp, ri, True, case["sets"])
            if case["block"] > 1:
                solver.set_block_preconditioner(case["block"], n // case["block"])
            return solver
        s["solver"] = _keep(_key(case), make)
        s["values"], s["b"] = _device(v), _device(b)
        s["x"] = torch.empty_like(s["b"])
        s["method"] = native.SOLVER_CG if case["method"] == "cg" else native.SOLVER_BICGSTAB
    else:
        s["X"], s["y"], s["p"] = _samples(case, rng)
        s["net"] = _keep(_key(case), lambda: native.MLP(case["features"], case["hidden"], 0))
    return s


def run(s):
    lib = native.symgb()
    if s["what"] == "assemble":
        u = s["unit"]
        if "out" not in s:
            for i, a in enumerate(s["inputs"]):
                u.set_arg(i, a)
            u.run()
            return u.get_result(0)
        for i, a in enumerate(s["inputs"]):
            native.check(lib.symgb_set_arg_sets_device(u.handle, C.c_void_p(a.data_ptr()), i))
        native.check(lib.symgb_run_async(u.handle))
        native.check(lib.symgb_get_result_sets_device(u.handle, C.c_void_p(s["out"].data_ptr()), 0))
        return s["out"]
    if s["what"] == "batch":
        for u, ins in zip(s["units"], s["inputs"]):
            for i, a in enumerate(ins):
                native.check(lib.symgb_set_arg_sets_device(u.handle, C.c_void_p(a.data_ptr()), i))
        native.check(lib.symgb_batch_run_async(s["batch"], C.c_void_p(_stream().cuda_stream)))
        for u, out in zip(s["units"], s["out"]):
            native.check(lib.symgb_get_result_sets_device(u.handle, C.c_void_p(out.data_ptr()), 0))
        return s["out"]
    if s["what"] == "solve":
        _, residual = s["solver"].solve(s["values"], s["b"], s["x"], tol=TOLERANCE, max_iter=2000, method=s["method"],
                                        stream=_stream())
        if not residual <= TOLERANCE:
            raise RuntimeError(f"solve stopped at {residual}")
        return s["x"]
    s["net"].set_params(s["p"])
    loss = s["net"].train(s["X"], s["y"], s["case"]["epochs"], LEARNING_RATE)
    return {"weights": s["net"].params(), "loss": np.float32(loss)}


# ---------------------------------------------------------------- work and exact values

_OPS = {3, 4, 5, 6, 7, 23, 26}  # add, multiply, multiply by constants, divide, root, negate, reciprocal


def _template(kernel):
    """The template's nodes in post-order: (op, child count, a, b, value)."""
    return [(n.op, n.nchild, n.a, n.b, n.value) for n in (kernel.nodes[j] for j in range(kernel.num_nodes))]


def _plan_work(plan, size, sets):
    w = _plan(plan, size)
    d = w.plan.contents
    flops = 0
    for k in range(d.num_kernels):
        kd = d.kernels[k]
        per = sum((c - 1 if op in (3, 4, 5) else 1) for op, c, *_ in _template(kd) if op in _OPS)
        flops += per * int(kd.num_instances)
    io = sum(a.size for a in w.inputs) + w.out_index_data.size
    return {"bytes": sets * 8 * io + 4 * w.index_data.size + 4 * w.out_index_data.size + 8 * w.const_data.size,
            "flops": sets * flops}


def work(case):
    if case["what"] == "assemble":
        return _plan_work(case["plan"], case["size"], case["sets"])
    if case["what"] == "batch":
        parts = [_plan_work("cloth", side, sets) for side, sets in _batch_members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if case["what"] == "solve":
        # values and right-hand sides read, solutions written; one product with
        # the matrix at the least
        n, cp, ri, ci = _keep(("pattern", case["side"]), lambda: _cloth_pattern(case["side"]))
        full = 2 * ri.size - n
        return {"bytes": case["sets"] * 8 * (ri.size + 2 * n) + 4 * ri.size, "flops": 2 * case["sets"] * full}
    n, f, h, e = (case[k] for k in ("samples", "features", "hidden", "epochs"))
    params = f * h + h * h + 3 * h + 1
    return {"bytes": 4 * (n * (f + 1) + 2 * params), "flops": e * n * (4 * f * h + 6 * h * h + 6 * h)}


def _evaluate(w, inputs):
    """Outputs of a plan in plain NumPy double arithmetic, one operation at a
    time: inputs [sets, length] per container -> [sets, outputs]."""
    d = w.plan.contents
    sets = inputs[0].shape[0]
    x = np.zeros((int(d.num_total_memory), sets))
    for i, a in enumerate(inputs):
        x[int(d.arg_start[i]):int(d.arg_start[i]) + a.shape[1]] = a.T
    for k in range(d.num_kernels):
        kd = d.kernels[k]
        n = int(kd.num_instances)
        if not n:
            continue
        access = [(kd.access[2 * a], kd.access[2 * a + 1]) for a in range(kd.num_access)]
        local, stack, y = {}, [], {}
        for op, c, a, b, value in _template(kd):
            kids = stack[len(stack) - c:] if c else []
            del stack[len(stack) - c:]
            if op == 1:
                v = value
            elif op == 2 and b == -3:
                row, offset = access[a]
                at = int(kd.index_offset) + row * n
                v = x[w.index_data[at:at + n].astype(np.int64) + offset]
            elif op == 2 and b == -4:
                at = int(kd.constants_offset) + a * n
                v = w.const_data[at:at + n, None]
            elif op == 2:
                v = local.get(a, ("name", b, a)) if b == 253 else ("name", b, a)
            elif op in (3, 4, 5):
                v = kids[0]
                for q in kids[1:]:
                    v = v + q if op == 3 else v * q
            elif op == 6:
                v = kids[0] / kids[1]
            elif op == 7:
                v = np.sqrt(kids[0])
            elif op == 23:
                v = -kids[0]
            elif op == 26:
                v = 1.0 / kids[0]
            elif op == 24:  # local = expression
                local[kids[0][2]] = kids[1]
                v = None
            elif op == 18:  # output row = expression
                y[kids[0][2]] = kids[1]
                v = None
            elif op == 25:
                v = None
            else:
                raise ValueError(f"operation {op}")
            stack.append(v)
        for row, v in y.items():
            at = int(kd.output_offset) + row * n
            x[at:at + n] = v
    return np.ascontiguousarray(x[w.out_index_data.astype(np.int64)].T)


def _conjugate_gradient(case, v, b):
    """Solutions in double precision, iterated until the residual stops falling."""
    n, cp, ri, ci = _kept[("pattern", case["side"])]
    off = ri != ci
    rows = torch.from_numpy(np.concatenate([ri, ci[off]]).astype(np.int64))
    cols = torch.from_numpy(np.concatenate([ci, ri[off]]).astype(np.int64))
    out = []
    for s in range(case["sets"]):
        vals = torch.from_numpy(np.concatenate([v[s], v[s][off]]))
        A = torch.sparse_coo_tensor(torch.stack([rows, cols]), vals, (n, n)).coalesce().to_sparse_csr()
        inv = 1.0 / torch.from_numpy(v[s][~off][np.argsort(ci[~off])])
        rhs = torch.from_numpy(b[s])
        x = torch.zeros(n, dtype=torch.float64)
        for _ in range(2):  # the second pass solves for what the first left
            r = rhs - A @ x
            z = inv * r
            p, rz = z.clone(), r @ z
            stop = 1e-15 * rhs.norm()
            for _ in range(600):
                q = A @ p
                alpha = rz / (p @ q)
                x = x + alpha * p
                r = r - alpha * q
                if r.norm() <= stop:
                    break
                z = inv * r
                rz, old = r @ z, rz
                p = z + (rz / old) * p
        out.append(x.numpy())
    return np.stack(out)


def _train(case, X, y, p):
    """The epochs of Adam on the mean squared error, in double precision."""
    f, h = case["features"], case["hidden"]
    X, y, p = X.astype(np.float64), y.astype(np.float64), p.astype(np.float64)
    cuts = np.cumsum([f * h, h, h * h, h, h, 1])[:-1]

    def parts(q):
        a = np.split(q, cuts)
        return a[0].reshape(f, h), a[1], a[2].reshape(h, h), a[3], a[4], a[5]

    def forward(q):
        W1, b1, W2, b2, W3, b3 = parts(q)
        h1 = np.maximum(X @ W1 + b1, 0.0)
        h2 = np.maximum(h1 @ W2 + b2, 0.0)
        return h1, h2, h2 @ W3 + b3
    m, v = np.zeros_like(p), np.zeros_like(p)
    for t in range(1, case["epochs"] + 1):
        _, _, W2, _, W3, _ = parts(p)
        h1, h2, out = forward(p)
        d = 2.0 * (out - y) / len(y)
        d2 = np.outer(d, W3) * (h2 > 0)
        d1 = (d2 @ W2.T) * (h1 > 0)
        g = np.concatenate([(X.T @ d1).ravel(), d1.sum(0), (h1.T @ d2).ravel(), d2.sum(0), h2.T @ d, [d.sum()]])
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - LEARNING_RATE * (m / (1 - 0.9 ** t)) / (np.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    return {"weights": p, "loss": np.float64(np.mean((forward(p)[2] - y) ** 2))}


def exact(case, seed):
    rng = np.random.default_rng(seed)
    if case["what"] == "assemble":
        ins = _values(case["plan"], case["size"], case["sets"], rng)
        w = _plan(case["plan"], case["size"])
        step = max(1, int(2e7 // max(1, w.num_total_memory)))  # a few sets at a time
        out = np.concatenate([_evaluate(w, [a[k:k + step] for a in ins]) for k in range(0, case["sets"], step)])
        return out.ravel() if case["io"] == "host" else out
    if case["what"] == "batch":
        return [_evaluate(_plan("cloth", side), _values("cloth", side, sets, rng))
                for side, sets in _batch_members(case)]
    if case["what"] == "solve":
        v, b = _system(case, rng)
        return _conjugate_gradient(case, v, b)
    X, y, p = _samples(case, rng)
    return _train(case, X, y, p)
