"""The plain solve's coarse-level kernels (kutta_b200/csrc/cuda/coarse_rows.cu):
rows whose products a block forms together, the folded transfers and the small
levels in one block must give the thread-per-row kernels' values, so whole
solves must match the oracle as before; and one FMA must give the bits of the
reference's split product error wherever it is used for it."""
import numpy as np
import pytest

from kutta_b200 import harness
from kutta_b200 import linalg as L
from oracle import kutta_oracle as O

M = L.OperatorStructure.SymmetricMMatrix
f32 = np.float32


def _split_error(a, b, product):
    """Dekker's product error with the 4097 split, in float32 throughout."""
    ca, cb = f32(4097) * a, f32(4097) * b
    ah, bh = ca - (ca - a), cb - (cb - b)
    al, bl = a - ah, b - bh
    return ((ah * bh - product) + ah * bl + al * bh) + al * bl


@pytest.mark.parametrize("low, high", [(-96, -90), (-60, 60), (60, 126)])
def test_fma_error_equals_split_error_above_2_to_minus_96(low, high):
    """For |a b| >= 2^-96 and factors up to 1e30 both are the exact error: a b
    has 48 bits, so float64 holds the product and its difference exactly."""
    rng = np.random.default_rng(low + 200)
    n = 400_000
    exponent = rng.integers(low, high, n)
    share = rng.integers(-40, 41, n)
    ea = np.clip(exponent // 2 + share, -126, 99)
    eb = np.clip(exponent - ea, -126, 99)
    a = np.ldexp(rng.uniform(1, 2, n), ea).astype(f32) * rng.choice([f32(-1), f32(1)], n)
    b = np.ldexp(rng.uniform(1, 2, n), eb).astype(f32)
    with np.errstate(over="ignore", invalid="ignore"):
        product = a * b
        used = np.isfinite(product) & (np.abs(product) >= f32(2.0 ** -96)) & \
            (np.abs(a) <= f32(1e30)) & (np.abs(b) <= f32(1e30))
        a, b, product = a[used], b[used], product[used]
        split = _split_error(a, b, product)
    exact = a.astype(np.float64) * b.astype(np.float64) - product.astype(np.float64)
    assert len(a) > n // 8
    assert np.array_equal(exact.astype(f32).astype(np.float64), exact)  # one FMA returns it
    assert np.array_equal(split, exact.astype(f32))


def _hub(n, degree, hubs, seed):
    """An M-matrix with a few rows of `degree` entries among rows of 3 to 6."""
    rng = np.random.default_rng(seed)
    pairs = {(i, i + 1) for i in range(n - 1)}
    for h in rng.choice(n, hubs, replace=False):
        for j in rng.choice(n, degree, replace=False):
            if h != j:
                pairs.add((min(h, j), max(h, j)))
    i, j = np.array(sorted(pairs)).T
    w = np.exp(rng.uniform(-3, 0, len(i))).astype(f32).astype(np.float64)
    row = np.concatenate([i, j, np.arange(n)])
    col = np.concatenate([j, i, np.arange(n)])
    total = np.bincount(np.concatenate([i, j]), np.concatenate([w, w]), n) * 1.001 + 1e-3
    diagonal = np.nextafter(total.astype(f32), f32(np.inf)).astype(np.float64)
    val = np.concatenate([-w, -w, diagonal])
    order = np.lexsort((col, row))
    row, col, val = row[order], col[order].astype(np.int32), val[order]
    row_ptr = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.int32)
    diag = np.nonzero(row == col)[0].astype(np.int32)
    return harness.HostSystem(row_ptr, col, diag, val, rng.standard_normal(n).astype(f32))


def _long_rows(n, length, seed):
    """An M-matrix of rows of about `length` entries."""
    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), length // 2)
    j = (i + rng.integers(1, n, len(i))) % n
    pairs = np.unique(np.minimum(i, j).astype(np.int64) * n + np.maximum(i, j))
    i, j = pairs // n, pairs % n
    w = rng.uniform(0.1, 1, len(i)).astype(f32).astype(np.float64)
    total = np.bincount(np.concatenate([i, j]), np.concatenate([w, w]), n) * 1.01 + 1e-3
    row = np.concatenate([i, j, np.arange(n)])
    col = np.concatenate([j, i, np.arange(n)])
    val = np.concatenate([-w, -w, np.nextafter(total.astype(f32), f32(np.inf))])
    order = np.lexsort((col, row))
    row, col, val = row[order], col[order].astype(np.int32), val[order].astype(np.float64)
    row_ptr = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.int32)
    diag = np.nonzero(row == col)[0].astype(np.int32)
    return harness.HostSystem(row_ptr, col, diag, val, rng.standard_normal(n).astype(f32))


CASES = {
    # Rows at and around a block's 32, 64 and 128, and one small level only.
    **{f"poisson{n}": lambda n=n: harness.poisson(n, 1) for n in (25, 33, 64, 65, 129, 257)},
    "poisson2d": lambda: harness.poisson(47, 43, 1, 100.0),
    # A smallest level too large for one block, and two that fit one.
    "hex": lambda: harness.box_system(27, 23, 26, tet=False, seed=4),
    "tet": lambda: harness.box_system(13, 17, 11, tet=True, seed=5),
    # Rows longer than what a block stages at once (1,024 and 2,048 entries).
    "hub_small": lambda: _hub(3_000, 1_400, 3, 1),
    "hub_large": lambda: _hub(20_000, 5_000, 4, 2),
    # Many long rows in a block: formed by the block (150), a thread per row (400).
    **{f"rows{k}": lambda k=k: _long_rows(1_500, k, 3) for k in (150, 400)},
}


# (system, coarse_rows, the rows and entries of some levels below the fine one).
ONE_BLOCK = {
    # The most rows a level in one block has, and one more; on the way down levels
    # of 256, 32 and 4 rows, or of 257, 33 and 5.
    "rows2048": (lambda: harness.poisson(16384, 1), 24, {1: (2048, 6142), 3: (32, 94)}),
    "rows2049": (lambda: harness.poisson(16392, 1), 24, {1: (2049, 6145), 3: (33, 97)}),
    # Coarsest levels about 24 rows, up to which a launch of its own takes the
    # coarsest, and 32, up to which a warp of the one block does.
    **{f"coarsest{c}": (lambda c=c: harness.poisson(8 * c, 1), c, {1: (c, 3 * c - 2)})
       for c in (24, 25, 32, 33)},
    # Two tet levels below and above 16,384 entries, the most one in a block has.
    "entries11452": (lambda: harness.box_system(14, 14, 12, tet=True, seed=5), 24,
                     {2: (1384, 11452), 3: (988, 6352)}),
    "entries16696": (lambda: harness.box_system(16, 15, 14, tet=True, seed=5), 24,
                     {2: (1984, 16696), 3: (1426, 9532)}),
}


@pytest.mark.gpu
@pytest.mark.parametrize("post", [3, 1])
@pytest.mark.parametrize("name", ONE_BLOCK)
def test_one_block_edges_match_oracle(cuda, name, post):
    """At the limits of the levels that run in one block, AMG-BiCGStab (whose
    sweeps down and up may differ) as below."""
    import torch
    make, coarse_rows, sizes = ONE_BLOCK[name]
    s = make()
    a = L.upload(s)
    solver = L.make_amg_solver(L.SolverKind.AmgBicgstab, s, L.AmgOptions(
        pre_sweeps=3, post_sweeps=post, coarse_rows=coarse_rows))
    solver.refresh(a)
    levels = solver.levels()
    for k, (rows, entries) in sizes.items():
        assert (levels[k][0], len(levels[k][2])) == (rows, entries), [lv[0] for lv in levels]
    x = torch.zeros(s.n, device="cuda")
    b = s.b.astype(f32)
    st = solver.solve(a, x, torch.from_numpy(b).cuda(), L.SolveControl(1e-4, 1e-38, 200))
    o = O.solve(s, O.AMG_BICGSTAB, b=b, rel_tol=1e-4, abs_tol=1e-38, max_iter=200,
                opts=O.options(O.AMG_BICGSTAB, pre_sweeps=3, post_sweeps=post,
                               coarse_rows=coarse_rows))
    got = x.cpu().numpy().astype(np.float64)
    assert (st.iterations, st.converged) == (o.iterations, o.converged)
    assert np.linalg.norm(got - o.x) <= 1e-5 * np.linalg.norm(o.x.astype(np.float64))


@pytest.mark.gpu
@pytest.mark.parametrize("point", [False, True], ids=["", "point"])
@pytest.mark.parametrize("name", CASES)
def test_solve_matches_oracle(cuda, name, point):
    """point: a single source, whose iterates are zero or tiny far from it, so
    that products fall below 2^-96, where the split itself runs. x within
    relative 1e-5 and equal iterations, as the solver parity tests require (the
    FP64 reductions alone may round otherwise)."""
    import torch
    s = CASES[name]()
    b = s.b.astype(f32)
    if point:
        b = np.zeros(s.n, f32)
        b[s.n // 3] = 1
    a = L.upload(s)
    solver = L.make_amg_solver(L.SolverKind.AmgPcg, s, L.AmgOptions(structure=M, pre_sweeps=3,
                                                                    post_sweeps=3))
    solver.refresh(a)
    x = torch.zeros(s.n, device="cuda")
    st = solver.solve(a, x, torch.from_numpy(b).cuda(), L.SolveControl(1e-4, 1e-38, 200))
    o = O.solve(s, O.AMG_PCG, m_matrix=True, b=b, rel_tol=1e-4, abs_tol=1e-38, max_iter=200,
                opts=O.options(O.AMG_PCG, pre_sweeps=3, post_sweeps=3, m_matrix=True))
    got = x.cpu().numpy().astype(np.float64)
    assert (st.iterations, st.converged) == (o.iterations, o.converged)
    assert np.linalg.norm(got - o.x) <= 1e-5 * np.linalg.norm(o.x.astype(np.float64))


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-32, 1e32])
def test_solve_beyond_the_split_guard(cuda, scale):
    """Entries or iterates above 1e30, where the reference's product error is
    zero: the same iterations as the oracle and x as above."""
    import torch
    s = harness.poisson(47, 43)
    s.val = (s.val * scale).astype(f32).astype(np.float64)
    b = np.random.default_rng(1).standard_normal(s.n).astype(f32)
    a = L.upload(s)
    solver = L.make_amg_solver(L.SolverKind.AmgPcg, s, L.AmgOptions(pre_sweeps=2, post_sweeps=2))
    solver.refresh(a)
    x = torch.zeros(s.n, device="cuda")
    st = solver.solve(a, x, torch.from_numpy(b).cuda(), L.SolveControl(1e-4, 1e-38, 200))
    o = O.solve(s, O.AMG_PCG, b=b, rel_tol=1e-4, abs_tol=1e-38, max_iter=200,
                opts=O.options(O.AMG_PCG, pre_sweeps=2, post_sweeps=2))
    got = x.cpu().numpy().astype(np.float64)
    assert (st.iterations, st.converged) == (o.iterations, o.converged)
    assert np.linalg.norm(got - o.x) <= 1e-5 * np.linalg.norm(o.x.astype(np.float64))


@pytest.mark.gpu
def test_updates_queued_past_the_end_are_skipped(cuda):
    """Updates that a batch still queues after the one that converged load their
    operators ahead, but form no products: on 1,572,864 tets such an update costs
    half of a running one, and three quarters where the sweeps are worked out."""
    import time
    import torch
    s = harness.box_system(64, 64, 64, tet=True, seed=1)
    a = L.upload(s)
    b = torch.from_numpy(s.b).cuda()

    def first_solve(interval):
        times, iterations = [], 0
        for _ in range(4):
            solver = L.make_amg_solver(L.SolverKind.AmgPcg, s, L.AmgOptions(
                structure=M, pre_sweeps=2, post_sweeps=2))
            solver.refresh(a)
            x = torch.zeros(s.n, device="cuda")
            torch.cuda.synchronize()
            start = time.perf_counter()
            st = solver.solve(a, x, b, L.SolveControl(1e-3, 1e-30, 500, interval))
            torch.cuda.synchronize()
            times.append(time.perf_counter() - start)
            assert st.converged and iterations in (0, st.iterations)
            iterations = st.iterations
        return min(times), iterations

    count = first_solve(1)[1]
    exact, same = first_solve(count)
    longer, again = first_solve(count + 40)
    assert same == again == count
    assert (longer - exact) / 40 < 0.62 * exact / count


@pytest.mark.gpu
@pytest.mark.parametrize("sides", [(200, 180, 1), (60, 60, 60)])
def test_general_refresh(cuda, sides):
    """A refresh without the M-matrix diagonal, with the first coarse level below and
    above 131,072 entries, where its diagonals are summed apart: the oracle's values
    bit for bit, in two launches a level and one for the levels in one block."""
    s = harness.poisson(*sides)
    a = L.upload(s)
    solver = L.make_amg_solver(L.SolverKind.AmgPcg, s, L.AmgOptions())
    solver.refresh(a)
    launches = L.kernel_launches()
    solver.refresh(a)
    launches = L.kernel_launches() - launches
    levels = solver.levels()
    assert launches <= 2 * len(levels)
    assert (len(levels[1][2]) > 1 << 17) == (sides[2] > 1)
    o = O.Solver(s, O.options(O.AMG_PCG))
    o.refresh(s.val.astype(f32))
    want = o.levels()
    for k, (got, ref) in enumerate(zip(levels, want, strict=True)):
        assert np.array_equal(got[4].view(np.uint32), ref["l1"].view(np.uint32)), k
        if k > 0:
            assert np.array_equal(got[3].view(np.uint32), ref["val"].view(np.uint32)), k


@pytest.mark.gpu
def test_levels_of_long_rows_are_not_slower_than_a_thread_per_row(cuda):
    """2,000 rows of some 480 entries, where a block would add the entries of a few
    rows at a time: a sweep of the solve takes no more than 1.3 times the sweep that
    amg_smooth launches, a thread per row (167 against 99 us when a block did)."""
    import time
    import torch
    s = _long_rows(2_000, 480, 1)
    a = L.upload(s)
    b = torch.from_numpy(s.b).cuda()

    def best(run):
        times = []
        for _ in range(5):
            torch.cuda.synchronize()
            start = time.perf_counter()
            run()
            torch.cuda.synchronize()
            times.append(time.perf_counter() - start)
        return min(times)

    def solve(sweeps):
        solver = L.make_amg_solver(L.SolverKind.AmgPcg, s, L.AmgOptions(
            coarse_sweeps=sweeps, max_levels=1, setup=L.Setup.Host))
        solver.refresh(a)
        x = torch.zeros_like(b)
        return best(lambda: solver.solve(a, x.zero_(), b, L.SolveControl(1e-30, 1e-38, 1)))

    x, y, inverse = torch.zeros_like(b), torch.zeros_like(b), torch.ones_like(b)

    def direct():
        for _ in range(100):
            L.amg_smooth(a, x, b, inverse, y)

    assert (solve(300) - solve(100)) / 200 <= 1.3 * best(direct) / 100
