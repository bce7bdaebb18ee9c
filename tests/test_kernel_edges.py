"""Kernels at the sizes where they change over: assembly rows at and above what
a thread holds in registers, the dense inverse around its warps' and slices'
edges, mixed coarse rows with and without columns in 16-bit reach and above the
two-rows rule, and the learned stage's backward at ragged row counts."""
import numpy as np
import pytest

from kutta_b200 import harness
from kutta_b200 import linalg as L
from oracle import fv

pytestmark = pytest.mark.gpu
M = L.OperatorStructure.SymmetricMMatrix


def _bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def _random_rows(n, degree, seed):
    """A symmetric M-matrix whose rows have up to `degree` off-diagonals."""
    rng = np.random.default_rng(seed)
    load = np.zeros(n, int)
    pairs = set()
    for i in range(n - 1):
        for j in {i + 1, *rng.integers(0, n, degree)}:
            p = (min(i, j), max(i, j))
            if i != j and p not in pairs and load[i] < degree and load[j] < degree:
                pairs.add(p)
                load[[i, j]] += 1
    i, j = np.array(sorted(pairs)).T
    w = np.exp(rng.uniform(-3, 0, len(i))).astype(np.float32).astype(np.float64)
    row = np.concatenate([i, j, np.arange(n)])
    col = np.concatenate([j, i, np.arange(n)])
    total = np.bincount(np.concatenate([i, j]), np.concatenate([w, w]), n) * 1.01 + 1e-3
    val = np.concatenate([-w, -w, np.nextafter(total.astype(np.float32), np.float32(np.inf))])
    return _system(row, col, val, n, rng)


def _system(row, col, val, n, rng):
    order = np.lexsort((col, row))
    row, col, val = row[order], col[order].astype(np.int32), val[order]
    row_ptr = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.int32)
    diag = np.nonzero(row == col)[0].astype(np.int32)
    return harness.HostSystem(row_ptr, col, diag, val.astype(np.float64),
                              rng.standard_normal(n).astype(np.float32))


def _device_fv(c):
    import torch
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    return L.FvPressure(t(c.offsets), t(c.faces), t(c.sign), t(c.adjacent), t(c.entry),
                        t(c.coefficient), t(c.flux), int(c.reference))


@pytest.mark.parametrize("reference", [-1, 100])
@pytest.mark.parametrize("degree, duplicate", [(3, 0.0), (4, 0.3), (5, 0.1), (6, 0.2), (8, 0.0),
                                               (13, 0.2)])
def test_assembly_rows_match_oracle_and_refresh(cuda, degree, duplicate, reference):
    """Faces below, at and above six per row, some sharing an entry, some
    entries without a face (they keep their value), some faces naming the
    diagonal: bit for bit the oracle's
    values, and with the refresh fused the separate refresh's levels."""
    import torch
    s = _random_rows(3000, degree, degree)
    c = harness.fv_faces(s.row_ptr, s.col, s.diag, seed=3, duplicate=duplicate, boundary=1.0,
                         reference=reference)
    # Every 50th internal face becomes a wall face of both its cells, so that
    # their entries may be left without one.
    slots = np.isin(c.faces, np.arange(0, c.internal, 50))
    c.adjacent[slots] = -1
    # A few others lie between a cell and itself (one layer of a periodic mesh).
    own = np.isin(c.faces, np.arange(7, c.internal, 90))
    cell = np.repeat(np.arange(s.n), np.diff(c.offsets))[own]
    c.adjacent[own] = cell
    c.entry[own] = s.diag[cell]
    start = s.val.astype(np.float32)
    v, r = start.copy(), np.zeros(s.n, np.float32)
    fv.oracle_assemble(c, v, r)
    a = L.upload(s)
    rhs = torch.zeros(s.n, device="cuda")
    L.fv_pressure_assemble(a, _device_fv(c), rhs)
    assert np.array_equal(_bits(a.val.cpu().numpy()), _bits(v))
    assert np.array_equal(_bits(rhs.cpu().numpy()), _bits(r))
    levels = []
    for fused in (False, True):
        a = L.upload(s)
        solver = L.make_amg_solver(L.SolverKind.AmgPcg, s, L.AmgOptions(structure=M))
        rhs = torch.zeros(s.n, device="cuda")
        if fused:
            solver.assemble_refresh(a, _device_fv(c), rhs)
        else:
            L.fv_pressure_assemble(a, _device_fv(c), rhs)
            solver.refresh(a)
        levels.append([a.val.cpu().numpy(), rhs.cpu().numpy(),
                       *(x for lv in solver.levels() for x in lv[3:5])])
        x = torch.zeros(s.n, device="cuda")
        solver.solve(a, x, rhs, L.SolveControl(1e-5, 1e-30, 300))
        levels[-1].append(x.cpu().numpy())  # reads the packed rows
    for one, two in zip(*levels):
        assert np.array_equal(_bits(one), _bits(two))


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 111, 112])
def test_dense_inverse_edges(cuda, n):
    """Against numpy in FP64: |error| <= n eps cond |inverse| to first order for
    an elimination without pivoting on an SPD matrix; 8 n eps cond allows for the
    products' own rounding."""
    import torch
    rng = np.random.default_rng(n)
    q = rng.standard_normal((n, n))
    dense = (q @ q.T / n + np.diag(rng.uniform(0.5, 2.0, n))).astype(np.float32).astype(np.float64)
    dense = np.tril(dense) + np.tril(dense, -1).T
    i, j = np.indices((n, n)).reshape(2, -1)
    a = L.upload(_system(i, j, dense.ravel(), n, rng))
    inv = torch.empty(n * n, dtype=torch.float64, device="cuda")
    flag = torch.full((1,), 7.0, dtype=torch.float64, device="cuda")
    L.dense_inverse(a, inv, flag)
    got, want = inv.cpu().numpy().reshape(n, n), np.linalg.inv(dense)
    assert flag.item() == 0.0
    bound = 8 * n * np.finfo(float).eps * np.linalg.cond(dense)
    assert np.max(np.abs(got - want)) <= bound * np.max(np.abs(want))


def _cholesky_fails(dense):
    """Whether a pivot of the FP64 Cholesky factor is not positive, each element
    updated by one FMA per step (the exact rational value rounded once)."""
    import math
    from fractions import Fraction
    n, fails = len(dense), False
    lower = dense.tolist()
    for k in range(n):
        d = lower[k][k]
        fails = fails or not d > 0
        root = math.sqrt(d) if d > 0 else 1.0
        column = [0.0] * (k + 1) + [lower[i][k] / root for i in range(k + 1, n)]
        exact = [Fraction(c) for c in column]
        for i in range(k + 1, n):
            for j in range(k + 1, i + 1):
                if column[i] and column[j]:
                    lower[i][j] = float(Fraction(lower[i][j]) - exact[i] * exact[j])
    return fails


@pytest.mark.parametrize("sides", [(3, 1), (18, 1), (2, 3), (3, 4), (4, 5), (5, 6), (6, 7), (7, 8),
                                   (8, 9), (9, 10), (4, 4, 4), (6, 4, 4), (7, 5, 3)])
@pytest.mark.parametrize("random", [False, True])
def test_dense_inverse_flags_singular_operators_by_the_factor(cuda, sides, random):
    """Neumann Laplacians, singular but for rounding: whether one is refused as not
    SPD follows the sign of the last pivot in the Cholesky factor."""
    import torch
    s = harness.poisson(*sides, *[1] * (4 - len(sides)), random, True)
    a = L.upload(s)
    inv = torch.empty(s.n * s.n, dtype=torch.float64, device="cuda")
    flag = torch.full((1,), 7.0, dtype=torch.float64, device="cuda")
    L.dense_inverse(a, inv, flag)
    dense = np.zeros((s.n, s.n))
    dense[np.repeat(np.arange(s.n), np.diff(s.row_ptr)), s.col] = s.val.astype(np.float32)
    assert flag.item() == float(_cholesky_fails(dense))


def _shuffled(s, seed):
    import scipy.sparse as sp
    rng = np.random.default_rng(seed)
    order = rng.permutation(s.n)
    A = sp.csr_matrix((s.val, s.col, s.row_ptr), shape=(s.n, s.n))[order][:, order].tocoo()
    return _system(A.row, A.col, A.data, s.n, rng)


@pytest.mark.parametrize("kind", ["pcg", "bicg"])
@pytest.mark.parametrize("name, make", [
    ("offset32767", lambda: harness.poisson(32767, 3)),
    ("offset32768", lambda: harness.poisson(32768, 3)),
    ("shuffled", lambda: _shuffled(harness.poisson(290, 230), 2)),
])
def test_plain_rows_with_near_and_far_columns(cuda, name, make, kind):
    """Levels read by a thread per row (more than 65,536 rows), with all columns
    within 16 bits of their row and without: whole solves against the oracle, x
    within relative 1e-5 and equal iterations, as the solver parity tests require."""
    import torch
    from oracle import kutta_oracle as O
    s = make()
    ours, theirs = ((L.SolverKind.AmgPcg, O.AMG_PCG) if kind == "pcg" else
                    (L.SolverKind.AmgBicgstab, O.AMG_BICGSTAB))
    a = L.upload(s)
    solver = L.make_amg_solver(ours, s, L.AmgOptions(pre_sweeps=2, post_sweeps=2))
    solver.refresh(a)
    b = np.random.default_rng(4).standard_normal(s.n).astype(np.float32)
    x = torch.zeros(s.n, device="cuda")
    st = solver.solve(a, x, torch.from_numpy(b).cuda(), L.SolveControl(1e-3, 1e-38, 60))
    o = O.solve(s, theirs, b=b, rel_tol=1e-3, abs_tol=1e-38, max_iter=60,
                opts=O.options(theirs, pre_sweeps=2, post_sweeps=2))
    got = x.cpu().numpy().astype(np.float64)
    assert (st.iterations, st.converged) == (o.iterations, o.converged)
    assert np.linalg.norm(got - o.x) <= 1e-5 * np.linalg.norm(o.x.astype(np.float64))


@pytest.mark.parametrize("sides", [(40, 33, 27), (96, 96, 72)])
@pytest.mark.parametrize("shuffled", [False, True], ids=["near", "far"])
def test_mixed_coarse_rows(cuda, sides, shuffled):
    """Coarse levels whose columns lie near their rows (value and column in one
    word) or, with shuffled cells and more than 32,767 coarse rows, far from
    them, on either side of 75,776 rows: the FP64 residual formed here meets the
    tolerance, in as many refinements either way (a wrong entry would stall)."""
    import scipy.sparse as sp
    import torch
    s = harness.box_system(*sides, tet=False, seed=6)
    A = sp.csr_matrix((s.val, s.col, s.row_ptr), shape=(s.n, s.n))
    rng = np.random.default_rng(1)
    if shuffled:
        order = rng.permutation(s.n)
        A = A[order][:, order].tocsr()
    A.sort_indices()
    row = np.repeat(np.arange(s.n), np.diff(A.indptr))
    t = harness.HostSystem(A.indptr.astype(np.int32), A.indices.astype(np.int32),
                           np.nonzero(row == A.indices)[0].astype(np.int32), A.data,
                           rng.standard_normal(s.n).astype(np.float32))
    a = L.upload(t)
    solver = L.make_mixed_solver(t)
    solver.refresh(a)
    x = torch.zeros(s.n, dtype=torch.float64, device="cuda")
    st = solver.solve(a, x, torch.from_numpy(t.b).cuda(), L.SolveControl(1e-9, 1e-30, 1000))
    b = t.b.astype(np.float64)
    assert st.converged and st.refinements <= 5
    assert np.linalg.norm(b - A @ x.cpu().numpy()) <= 1.0001e-9 * np.linalg.norm(b)


@pytest.mark.parametrize("cycle, sweeps", [(L.AmgCycle.V, 1), (L.AmgCycle.V, 2), (L.AmgCycle.K, 1),
                                           (L.AmgCycle.K, 3)], ids=["v1", "v2", "k1", "k3"])
@pytest.mark.parametrize("make, one_block", [
    # 62 rows below (no level in between); 125 + 15; 500 + 62; 1,024 and 1,025 rows,
    # of which the first fill the block; 1,125, 140 and 18.
    (lambda: harness.poisson(500, 1), False),
    *((lambda n=n: harness.poisson(n, 1), True) for n in (1000, 4000, 8192, 8200, 9000)),
    (lambda: harness.box_system(10, 10, 10, tet=True, seed=2), True),
    (lambda: harness.box_system(24, 22, 20, tet=False, seed=3), True),
    # Rows of up to 76 entries; more entries than shared memory holds.
    (lambda: _random_rows(3000, 6, 8), True),
    (lambda: _random_rows(7000, 9, 8), False),
], ids=["500", "1000", "4000", "8192", "8200", "9000", "tet", "hex", "hubs", "large"])
def test_small_levels_in_one_block(cuda, make, one_block, cycle, sweeps):
    """One application of the preconditioner with its smallest levels in one
    block against the same with the cluster launch and separate kernels
    (fused_coarse): the same steps in FP32, whose sums of a few tens of terms may
    run in another order, each rounding within 32 eps of its row's terms, and a
    cycle that contracts: 1e-5 relative."""
    import torch
    s = make()
    a = L.upload(s)
    b = torch.from_numpy(s.b).cuda()
    z = []
    for fused in (False, True):
        amg = L.AmgOptions(cycle=cycle, pre_sweeps=sweeps, post_sweeps=sweeps, structure=M)
        solver = L.make_mixed_solver(s, L.MixedOptions(amg=amg, fused_coarse=fused))
        solver.refresh(a)
        out = torch.zeros(s.n, device="cuda")
        solver.precondition(a, b, out)
        z.append(out.double().cpu().numpy())
        if not fused:
            assert ("in one block" in solver.describe()) == one_block, solver.describe()
    assert np.linalg.norm(z[0] - z[1]) <= 1e-5 * np.linalg.norm(z[1])


@pytest.mark.parametrize("n", [2, 7, 9, 31, 33, 127, 129, 1001, 4097])
def test_learned_gradient_at_ragged_sizes(cuda, n):
    """Row counts that leave a part of a thread's eight rows, a warp's or a
    128-row tile: the FP32 backward against the tensor-core one, whose BF16
    operands carry 8 bits (3e-2 of each block, as at full sizes), and its loss."""
    import scipy.sparse as sp
    import torch
    s = harness.poisson(n, 1)
    a = L.upload(s)
    g = L.LearnedStage(seed=5)
    g.bind(a)
    A = sp.csr_matrix((s.val, s.col, s.row_ptr), shape=(n, n))
    e = np.random.default_rng(n).standard_normal(n)
    t = torch.from_numpy((A @ e).astype(np.float32)).cuda()
    e = torch.from_numpy(e.astype(np.float32)).cuda()
    tc, loss_tc = g.gradient(t, e, tensor_cores=True)
    fp, loss_fp = g.gradient(t, e, tensor_cores=False)
    assert np.all(np.isfinite(fp)) and np.linalg.norm(fp) > 0
    assert loss_tc == pytest.approx(loss_fp, rel=1e-5, abs=1e-6)
    assert np.linalg.norm(tc - fp) <= 3e-2 * np.linalg.norm(fp)
