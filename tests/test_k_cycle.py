"""K-cycle solves against the same method in FP64: the flexible PCG with two
inner conjugate steps per coarse level (Solver::inner), on the hierarchy that the
solver holds."""
import numpy as np
import pytest
import scipy.sparse as sp

from kutta_b200 import harness
from kutta_b200 import linalg as L

pytestmark = pytest.mark.gpu


def _bf16_rows(v, row_ptr):
    """The values that the mixed solve's coarse rows hold: max |a_ij| times the
    BF16 rounding of a_ij over it (float operations)."""
    import torch
    row = np.repeat(np.arange(len(row_ptr) - 1), np.diff(row_ptr))
    scale = np.zeros(len(row_ptr) - 1, np.float32)
    np.maximum.at(scale, row, np.abs(v))
    scale[scale == 0] = 1
    share = v * (np.float32(1) / scale)[row]
    return scale[row].astype(np.float64) * torch.from_numpy(share).bfloat16().double().numpy()


class Model:
    """The cycle and its flexible PCG in FP64 on the solver's own levels; with
    `constant`, corrections and coarse right-hand sides are projected."""

    def __init__(self, solver, a, sweeps, k_levels=0, bf16=False, constant=False,
                 coarse_sweeps=32):
        self.sweeps, self.coarse_sweeps = sweeps, coarse_sweeps
        self.k_levels, self.constant = k_levels, constant
        self.second_steps = 0
        self.levels = []
        for k, (n, rp, cl, vl, l1, ag) in enumerate(solver.levels()):
            v = a.val.cpu().numpy() if k == 0 else _bf16_rows(vl, rp) if bf16 else vl
            A = sp.csr_matrix((v.astype(np.float64), cl, rp), shape=(n, n))
            self.levels.append((A, l1.astype(np.float64), ag))

    def project(self, v):
        return v - v.mean() if self.constant else v

    def smooth(self, k, b, x, sweeps):
        A, l1, _ = self.levels[k]
        for _ in range(sweeps):
            x = x + 2 / 3 * l1 * (b - A @ x)
        return x

    def cycle(self, k, b):
        A, _, ag = self.levels[k]
        x = np.zeros(A.shape[0])
        if k + 1 == len(self.levels):
            return self.project(self.smooth(k, b, x, self.coarse_sweeps))
        x = self.smooth(k, b, x, self.sweeps)
        nc = self.levels[k + 1][0].shape[0]
        at = ag >= 0
        rc = self.project(np.bincount(ag[at], (b - A @ x)[at], nc))
        inner = k + 2 < len(self.levels) and (self.k_levels == 0 or k < self.k_levels)
        xc = self.inner(k + 1, rc) if inner else self.cycle(k + 1, rc)
        x[at] += xc[ag[at]]
        return self.project(self.smooth(k, b, x, self.sweeps))

    def inner(self, k, b):
        A = self.levels[k][0]
        p = self.cycle(k, b)
        q = A @ p
        pq = p @ q
        alpha = b @ p / pq
        x, t = alpha * p, b - alpha * q
        if t @ t <= b @ b / 16:
            return x
        self.second_steps += 1
        z = self.cycle(k, t)
        p = z - (z @ q) / pq * p
        q = A @ p
        return x + t @ p / (p @ q) * p

    def solve(self, b, rel_tol, max_iter):
        A = self.levels[0][0]
        x, r = np.zeros(len(b)), b.copy()
        z = self.cycle(0, r)
        p, rho = z.copy(), r @ z
        for k in range(1, max_iter + 1):
            q = A @ p
            alpha = rho / (p @ q)
            x, r = x + alpha * p, r - alpha * q
            if np.linalg.norm(r) <= rel_tol * np.linalg.norm(b):
                return k, x
            z = self.cycle(0, r)
            p = z - alpha * (z @ q) / rho * p
            rho = r @ z
        return max_iter, x


# 65,536 rows is where the fine level's row kernels change.
@pytest.mark.parametrize("sweeps", [1, 2, 3])
@pytest.mark.parametrize("make, max_levels", [
    (lambda: harness.poisson(24, 24, 24), 2), (lambda: harness.poisson(24, 24, 24), 24),
    (lambda: harness.poisson(40, 40, 40), 24), (lambda: harness.poisson(64, 32, 32), 24),
    (lambda: harness.poisson(41, 41, 41), 24),
    (lambda: harness.box_system(14, 13, 12, tet=True, seed=3), 24),
], ids=["24_two_grid", "24", "40", "65536", "41", "tet"])
def test_plain_k_cycle_follows_fp64(cuda, make, max_levels, sweeps):
    """As many iterations as in FP64 and x within relative 1e-5, as the solver
    parity tests require (FP32 vectors, compensated row sums, FP64 dots)."""
    import torch
    s = make()
    a = L.upload(s)
    solver = L.make_amg_solver(L.SolverKind.AmgPcg, s, L.AmgOptions(
        cycle=L.AmgCycle.K, pre_sweeps=sweeps, post_sweeps=sweeps, max_levels=max_levels))
    solver.refresh(a)
    b = np.random.default_rng(5).standard_normal(s.n).astype(np.float32)
    x = torch.zeros(s.n, device="cuda")
    st = solver.solve(a, x, torch.from_numpy(b).cuda(), L.SolveControl(1e-4, 1e-30, 300))
    model = Model(solver, a, sweeps)
    iterations, want = model.solve(b.astype(np.float64), 1e-4, 300)
    got = x.cpu().numpy().astype(np.float64)
    assert st.converged and st.iterations == iterations
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("k_levels", [1, 0], ids=["k_level1", "k_all"])
@pytest.mark.parametrize("sweeps", [1, 2])
@pytest.mark.parametrize("sides", [(17, 17, 17), (33, 21, 30)])
def test_mixed_k_cycle_with_constant_nullspace(cuda, sides, sweeps, k_levels):
    """One application of the preconditioner on a Neumann problem, whose inner
    steps' products take the projected corrections: FP32 against FP64 on the same
    BF16 rows, each of some twenty passes rounding to 6e-8. (Sides whose singular
    coarsest operator has a positive last pivot, so that it is not refused.)"""
    import torch
    s = harness.poisson(*sides, 1, False, True)
    a = L.upload(s)
    options = dict(cycle=L.AmgCycle.K, pre_sweeps=sweeps, post_sweeps=sweeps,
                   nullspace=L.NullSpace.Constant)
    solver = L.make_mixed_solver(s, L.MixedOptions(
        amg=L.AmgOptions(**options), k_cycle_levels=k_levels, absorb_singletons=False))
    solver.refresh(a)
    assert "smoothed instead of its dense inverse" in solver.describe()
    b = np.random.default_rng(3).standard_normal(s.n).astype(np.float32)
    z = torch.zeros(s.n, device="cuda")
    solver.precondition(a, torch.from_numpy(b).cuda(), z)
    # The same hierarchy, whose levels can be read back.
    plain = L.make_amg_solver(L.SolverKind.AmgPcg, s, L.AmgOptions(coarse_rows=112, **options))
    plain.refresh(a)
    model = Model(plain, a, sweeps, k_levels, bf16=True, constant=True)
    want = model.cycle(0, b.astype(np.float64))
    err = np.linalg.norm(z.cpu().numpy() - want) / np.linalg.norm(want)
    assert (model.second_steps == 1) == (k_levels == 1 or sides[0] == 17)
    assert err <= 1e-6
