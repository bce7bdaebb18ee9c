"""The Coupled solve's coarse-level kernels (kutta_b200/csrc/cuda/coupled_coarse.cu)
on boxes whose levels reach both launch shapes and rows of a hundred entries:
row kernels and Galerkin sums bit for bit against numpy restatements of the
reference's order, on the operators that the device assembled."""
import numpy as np
import pytest

from kutta_b200 import coupled_harness as H
from kutta_b200 import linalg as L
from oracle import coupled as O

pytestmark = pytest.mark.gpu
f32 = np.float32

BOXES = {
    # More than 16,384 rows on level 1, a ragged last block on every level.
    "hex": lambda: H.box_hex(53, 51, 49),
    # Hub rows on the small levels, and levels at the one-block tail's edges.
    "tet": lambda: H.box_tet(12, 11, 9),
}


def bits(a):
    return np.ascontiguousarray(a, f32).view(np.uint32)


def _solve(mesh, fields, reference=-1, options=None, max_iter=20):
    import torch
    dev = {k: torch.from_numpy(v).cuda() if isinstance(v, np.ndarray) else v
           for k, v in fields.items()}
    s = L.CoupledSolver(mesh, reference, options or L.CoupledOptions())
    rows, diag = (torch.from_numpy(mesh[k]).cuda() for k in ("pattern_row_ptr", "pattern_diag"))
    for k, c in enumerate("uvw"):
        s.capture_diagonal(k, rows, diag, dev["momentum_" + c], dev["physical_" + c])
    s.solve(dev, L.SolveControl(0.1, 1e-12, max_iter))
    return s


def _solved(name):
    mesh = BOXES[name]()
    return _solve(mesh, H.flow_fields(mesh, 3))


@pytest.mark.parametrize("name", BOXES)
def test_level_rows_match_oracle(cuda, name):
    import torch
    s = _solved(name)
    omega = L.CoupledOptions().smoother_damping
    rng = np.random.default_rng(5)
    for k in range(1, s.levels()):
        lv = s.level(k)
        n = len(lv["diag"])
        x, b = (rng.standard_normal(4 * n).astype(f32) for _ in range(2))
        dx, db = (torch.from_numpy(np.ascontiguousarray(v.reshape(4, n).T).reshape(-1)).cuda()
                  for v in (x, b))
        want = {"residual": (b - O.coarse_row(lv, x)).astype(f32),
                "smooth": O.coarse_smooth(lv, x, b, omega, False),
                "smooth_zero": O.coarse_smooth(lv, x, b, omega, True)}
        for op, w in want.items():
            y = torch.full((4 * n,), float("nan"), device="cuda")
            s.level_apply(k, op, dx, db, y)
            got = y.cpu().numpy().reshape(n, 4).T.reshape(-1)
            assert np.array_equal(bits(got), bits(w)), (k, op)


class Cycle:
    """The V-cycle on the oracle's row kernels, with the device's operators."""

    def __init__(self, s, mesh, fields, o):
        self.mesh, self.o = mesh, o
        self.wc = f32(fields["density"] * fields["velocity_scale"])
        self.cell, self.coefficient = s.copy("cell"), s.copy("coefficient")
        self.edge = O.fine_coefficients(mesh, self.cell, fields["viscosity"], fields["mass"],
                                        fields["face_weights"], self.wc)
        self.levels = [s.level(k) for k in range(1, s.levels())]

    def fine_row(self, x):
        return O.fine_row(self.mesh, self.cell, self.edge, self.coefficient, x, self.wc)

    def sweeps(self, k, x, b, count, first):
        for q in range(count):
            zero = first and q == 0
            if k == 0:
                x = O.fine_smooth(self.mesh, self.cell, self.edge, self.coefficient, x, b, self.wc,
                                  self.o.smoother_damping, zero)
            else:
                x = O.coarse_smooth(self.levels[k - 1], x, b, self.o.smoother_damping, zero)
        return x

    def __call__(self, b, k=0):
        if k == len(self.levels):
            return self.sweeps(k, None, b, self.o.coarsest_sweeps, True)
        n = len(b) // 4
        x = self.sweeps(k, None, b, self.o.pre_sweeps, True)
        r = b - (self.fine_row(x) if k == 0 else O.coarse_row(self.levels[k - 1], x))
        aggregate = self.levels[k]["aggregate"]
        members = np.argsort(aggregate, kind="stable").astype(np.int32)
        offsets = np.concatenate([[0], np.cumsum(np.bincount(aggregate))])
        c = self(O.restrict(offsets, members, r.astype(f32), n), k + 1).reshape(4, -1)
        x = (x.reshape(4, n) + c[:, aggregate]).reshape(-1)
        return self.sweeps(k, x, b, self.o.post_sweeps, False)


@pytest.mark.parametrize("tail", ["1", "0"], ids=["tail", "separate"])
@pytest.mark.parametrize("post", [0, 1, 2])
@pytest.mark.parametrize("name", BOXES)
def test_one_update_follows_the_oracle(cuda, name, post, tail, monkeypatch):
    """The first BiCGStab update with the whole V-cycle, its folded transfers and
    first sweeps among it, on a coarse level above 16,384 rows and those below: the
    cycle rounds as the oracle's, and FP64 dots give the two coefficients, so x
    differs by float roundings only."""
    monkeypatch.setenv("KUTTA_B200_COUPLED_TAIL", tail)
    mesh = BOXES[name]()
    fields, o = H.flow_fields(mesh, 3), L.CoupledOptions(post_sweeps=post)
    s = _solve(mesh, fields, options=o, max_iter=1)
    cycle = Cycle(s, mesh, fields, o)
    n = len(cycle.levels[0]["diag"])
    assert (n > 16384) == (name == "hex") and len(cycle.levels[1]["diag"]) < 16384
    r = s.copy("rhs")

    def dot(a, b):
        return a.astype(np.float64) @ b.astype(np.float64)

    z = cycle(r)
    v = cycle.fine_row(z)
    alpha = dot(r, r) / dot(r, v)
    sv = (r - f32(alpha) * v).astype(f32)
    zs = cycle(sv)
    t = cycle.fine_row(zs)
    want = alpha * z.astype(np.float64) + dot(t, sv) / dot(t, t) * zs
    assert np.linalg.norm(s.copy("x") - want) <= 1e-6 * np.linalg.norm(want)


def _add(sum_, error, value):
    """One term of the Neumaier sum that the reference's diagonals take."""
    total = f32(sum_ + value)
    if abs(sum_) >= abs(value):
        error = f32(error + f32(f32(sum_ - total) + value))
    else:
        error = f32(error + f32(f32(value - total) + sum_))
    return total, error


def test_galerkin_sums_match_their_order(cuda):
    """Level 2 from level 1 (fv_coupled.kern.h:490-524): off-diagonal entries
    are plain sums in member and entry order, the diagonal's ten compensated."""
    s = _solved("tet")
    f, c = s.level(1), s.level(2)
    agg = c["aggregate"]
    n, nc, fz, cz = len(f["diag"]), len(c["diag"]), len(f["cols"]), len(c["cols"])
    entry = np.concatenate([[f["a"], f["c"]], f["g"].reshape(3, fz), f["h"].reshape(3, fz)])
    want = np.zeros((8, cz), f32)
    momentum = np.zeros((3, nc), f32)
    where = [{int(c["cols"][e]): e for e in range(c["rows"][i], c["rows"][i + 1])}
             for i in range(nc)]
    for i in range(nc):
        sums = np.zeros(10, f32)
        errors = np.zeros(10, f32)
        for row in np.nonzero(agg == i)[0]:
            for k in range(3):
                sums[k], errors[k] = _add(sums[k], errors[k], f["d"][k * n + row])
            for j in range(f["rows"][row], f["rows"][row + 1]):
                target = int(agg[f["cols"][j]])
                if j == f["diag"][row] or target == i:
                    if j != f["diag"][row]:
                        for k in range(3):
                            sums[k], errors[k] = _add(sums[k], errors[k], entry[0, j])
                    for k in range(7):
                        sums[3 + k], errors[3 + k] = _add(sums[3 + k], errors[3 + k],
                                                          entry[1 + k, j])
                else:
                    want[:, where[i][target]] += entry[:, j]
        total = (sums + errors).astype(f32)
        momentum[:, i] = total[:3]
        want[1:, c["diag"][i]] = total[3:]
        want[0, c["diag"][i]] = 0
    got = np.concatenate([[c["a"], c["c"]], c["g"].reshape(3, cz), c["h"].reshape(3, cz)])
    assert np.array_equal(bits(got), bits(want))
    assert np.array_equal(bits(c["d"][:3 * nc]), bits(momentum.reshape(-1)))


def test_long_term_lists_change_no_bits(cuda, monkeypatch):
    """The Galerkin terms numbered in 64 bits, on every level."""
    want = _solved("tet")
    monkeypatch.setenv("KUTTA_B200_COUPLED_LONG_TERMS", "1")
    got = _solved("tet")
    for k in range(1, want.levels()):
        a, b = want.level(k), got.level(k)
        for key in a:
            assert np.array_equal(a[key], b[key]), (k, key)
    assert np.array_equal(bits(want.copy("x")), bits(got.copy("x")))


def _hub_mesh(n):
    """A closed ring of n cells, each with a face to one cell more: connectivity
    only, the cells' places random and the areas along the distances."""
    rng = np.random.default_rng(1)
    centroid = rng.uniform(-1, 1, (n + 1, 3))
    ring = np.arange(n - 1)
    owner = np.concatenate([ring, [0], np.arange(n)])
    neighbour = np.concatenate([ring + 1, [n - 1], np.full(n, n)])
    order = np.lexsort((neighbour, owner))
    owner, neighbour = owner[order], neighbour[order]
    d = centroid[neighbour] - centroid[owner]
    area = d / np.linalg.norm(d, axis=1)[:, None] * np.where(neighbour == n, 1e-7, 1e-3)[:, None]
    fc = 0.5 * (centroid[owner] + centroid[neighbour])
    return H._mesh_arrays(centroid, np.full(n + 1, 1e-6), owner, neighbour, area, fc,
                          np.zeros(0, np.int64))


@pytest.mark.parametrize("n", [500, 46_345])
def test_galerkin_operator_of_a_hub_cell(cuda, n):
    """One cell that borders all others makes the fine slots cells x cells: 60 GB
    and more than 2^31 of them at the larger size. The first coarse operator is the
    fine one between prolongation and restriction, whose float sums of up to n terms
    are within 1e-4 of each other's."""
    import torch
    if n > 1000 and torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("80 GB of device memory")
    mesh = _hub_mesh(n)
    s = _solve(mesh, H.flow_fields(mesh, 3, reference=0), reference=0, max_iter=2)
    coarse = s.level(1)
    nc = len(coarse["diag"])
    x = torch.randn(4 * nc, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    zero, product = torch.zeros_like(x), torch.zeros_like(x)
    s.level_apply(1, "residual", x, zero, product)
    fine = torch.zeros(4 * (n + 1), device="cuda")
    s.level_apply(1, "prolong", x, None, fine)
    y, want = torch.zeros_like(fine), torch.zeros_like(x)
    s.apply("spmv", fine, None, y)
    s.level_apply(1, "restrict", y, None, want)
    got, want = -product.view(-1, 4).double(), want.view(-1, 4).double()
    assert nc > 48 and torch.isfinite(got).all()
    for k in range(4):
        assert (got - want)[:, k].norm() <= 1e-4 * want[:, k].norm()
