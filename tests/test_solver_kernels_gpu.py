"""The solver's kernels at the edges of their thread layouts: set counts that
do and do not divide a block, several threads to a row (1, 2 and 4 sets), a
single row, rows without entries, lower-triangle and full patterns."""
import numpy as np
import pytest

from symboliclib_gb300 import native

pytestmark = pytest.mark.gpu


def pattern(n, density, lower, rng, diagonal=True):
    """CSC pattern of a random symmetric matrix (lower triangle or full)."""
    m = rng.random((n, n)) < density
    m = np.tril(m | m.T)
    np.fill_diagonal(m, diagonal)
    if not lower:
        m = m | m.T
    cp = np.concatenate([[0], np.cumsum(m.sum(0))])
    return cp, np.concatenate([np.flatnonzero(m[:, j]) for j in range(n)]).astype(np.int32)


def dense(n, cp, ri, v, lower):
    A = np.zeros((n, n))
    for j in range(n):
        A[ri[cp[j]:cp[j + 1]], j] = v[cp[j]:cp[j + 1]]
    return A + np.tril(A, -1).T if lower else A


@pytest.mark.parametrize("n", [1, 37, 400])
@pytest.mark.parametrize("sets", [1, 2, 3, 4, 5, 8, 33, 100, 129, 256])
@pytest.mark.parametrize("lower", [True, False])
def test_multiply(n, sets, lower):
    """|q - A p| <= (terms of a row) 2^-53 |A| |p| with room for either summation order."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n * 1000 + sets)
    cp, ri = pattern(n, 0.08, lower, rng, diagonal=n == 1)
    if not len(ri):
        return
    v, p = rng.standard_normal((sets, len(ri))), rng.standard_normal((sets, n))
    q = torch.full((sets, n), np.nan, dtype=torch.float64, device="cuda")
    native.SparseSolver(n, cp, ri, lower, sets).multiply(torch.from_numpy(v).cuda(), torch.from_numpy(p).cuda(), q)
    q = q.cpu().numpy()
    for s in {0, sets // 2, sets - 1}:
        A = dense(n, cp, ri, v[s], lower)
        assert np.all(np.abs(q[s] - A @ p[s]) <= 2 * n * 2.0 ** -53 * (np.abs(A) @ np.abs(p[s])))


@pytest.mark.parametrize("sets,n", [(3, 19456), (3, 19457), (3, 30001), (3, 38913), (5, 9728), (5, 9729), (5, 19456),
                                    (5, 19457), (7, 12345), (11, 5000), (33, 5003)])
def test_multiply_many_rows(sets, n):
    """Row counts around which a row's threads change; at most 9 terms a row, either summation order."""
    torch = pytest.importorskip("torch")
    sp = pytest.importorskip("scipy.sparse")
    rng = np.random.default_rng(n + sets)
    rows, cols = [np.arange(n)], [np.arange(n)]
    for shift in (1, 2, 77, 4999):
        i = np.flatnonzero(rng.random(n - shift) < 0.7)
        rows.append(i + shift)
        cols.append(i)
    m = sp.csc_matrix((np.ones(sum(map(len, rows))), (np.concatenate(rows), np.concatenate(cols))), (n, n))
    m.sort_indices()
    v, p = rng.standard_normal((sets, m.nnz)), rng.standard_normal((sets, n))
    q = torch.full((sets, n), np.nan, dtype=torch.float64, device="cuda")
    solver = native.SparseSolver(n, m.indptr.astype(np.int64), m.indices.astype(np.int32), True, sets)
    solver.multiply(torch.from_numpy(v).cuda(), torch.from_numpy(p).cuda(), q)
    q = q.cpu().numpy()
    for s in range(sets):
        m.data[:] = v[s]
        A = m + sp.tril(m, -1).T
        assert np.all(np.abs(q[s] - A @ p[s]) <= 2 * 9 * 2.0 ** -53 * (abs(A) @ np.abs(p[s])))


@pytest.mark.parametrize("method,block", [(native.SOLVER_CG, 1), (native.SOLVER_BICGSTAB, 1),
                                          (native.SOLVER_BICGSTAB, 2), (native.SOLVER_BICGSTAB, 4)])
@pytest.mark.parametrize("n,sets", [(4, 1), (36, 2), (36, 7), (400, 4), (400, 40), (20, 256)])
def test_solve_diagonally_dominant(n, sets, method, block):
    """Condition number at most 1.5 * 3 (Gershgorin discs around uneven
    diagonals within a factor 3, radius a fifth), residual 1e-12: the solution to 1e-11."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + sets)
    cp, ri = pattern(n, 0.1, True, rng)
    v = rng.uniform(-1.0, 1.0, (sets, len(ri)))
    col = np.repeat(np.arange(n), np.diff(cp))
    off = ri != col
    for s in range(sets):
        row = np.bincount(ri[off], np.abs(v[s, off]), n) + np.bincount(col[off], np.abs(v[s, off]), n)
        v[s, off] *= 0.2 / max(row.max(), 1.0) if off.any() else 1.0
        v[s, ~off] = rng.uniform(1.0, 3.0, n)
    b = rng.standard_normal((sets, n))
    solver = native.SparseSolver(n, cp, ri, True, sets)
    for stride in ([1] if block == 1 else [1, n // block]):
        if block > 1:
            solver.set_block_preconditioner(block, stride)
        x = torch.full((sets, n), np.nan, dtype=torch.float64, device="cuda")
        it, res = solver.solve(torch.from_numpy(v).cuda(), torch.from_numpy(b).cuda(), x, tol=1e-12, max_iter=64,
                               method=method)
        assert res <= 1e-12
        for s in {0, sets - 1}:
            ref = np.linalg.solve(dense(n, cp, ri, v[s], True), b[s])
            assert np.linalg.norm(x[s].cpu().numpy() - ref) <= 1e-11 * np.linalg.norm(ref)


@pytest.mark.parametrize("method", [native.SOLVER_CG, native.SOLVER_BICGSTAB])
@pytest.mark.parametrize("where", ["b nan", "b inf", "values nan", "b huge", "all"])
def test_systems_that_are_not_finite_are_not_reported_as_solved(method, where):
    """Beside them the other systems, one of them with b = 0, are solved to the
    tolerance, and nobody waits for what cannot converge."""
    torch = pytest.importorskip("torch")
    n, sets = 60, 5
    rng = np.random.default_rng(4)
    cp, ri = pattern(n, 0.1, True, rng)
    col = np.repeat(np.arange(n), np.diff(cp))
    v = rng.uniform(-1.0, 1.0, (sets, len(ri))) * 0.02
    v[:, ri == col] = rng.uniform(1.0, 3.0, (sets, n))
    b = rng.standard_normal((sets, n))
    b[3] = 0.0
    bad = list(range(sets)) if where == "all" else [1]
    for s in bad:
        if where == "values nan":
            v[s, 7] = np.nan
        elif where == "b huge":
            b[s] *= 1e200  # its square is beyond the double range
        else:
            b[s, 5] = np.inf if where == "b inf" else np.nan
    solver = native.SparseSolver(n, cp, ri, True, sets)
    x = torch.full((sets, n), 7.0, dtype=torch.float64, device="cuda")
    it, res = solver.solve(torch.from_numpy(v).cuda(), torch.from_numpy(b).cuda(), x, tol=1e-12, max_iter=640,
                           method=method)
    assert res == np.inf and it <= 64
    for s in set(range(sets)) - set(bad):
        ref = np.linalg.solve(dense(n, cp, ri, v[s], True), b[s])
        assert np.linalg.norm(x[s].cpu().numpy() - ref) <= 1e-11 * np.linalg.norm(ref)


@pytest.mark.parametrize("sets", [1, 4])
def test_matrices_without_entries_are_refused(sets):
    torch = pytest.importorskip("torch")
    solver = native.SparseSolver(3, np.zeros(4, np.int64), np.zeros(0, np.int32), False, sets)
    v, b = torch.zeros(1, dtype=torch.float64, device="cuda"), torch.ones((sets, 3), dtype=torch.float64, device="cuda")
    with pytest.raises(RuntimeError):
        solver.multiply(v, b, torch.empty_like(b))
    for method in (native.SOLVER_CG, native.SOLVER_BICGSTAB):
        with pytest.raises(RuntimeError):
            solver.solve(v, b, torch.empty_like(b), tol=1e-12, max_iter=16, method=method)
