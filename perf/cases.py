"""The work that a flow solver has this library do, as cases to be timed.

A SIMPLE-type outer iteration assembles the pressure-correction matrix on the
device, refreshes the AMG hierarchy that was built once for the mesh, solves
from zero and corrects fluxes and velocities; a Coupled iteration hands the
block solver its momentum rows and takes the update. The setup (hierarchy from
the pattern) happens once per mesh, so it belongs to `prepare`; every value
change pays for the refresh, so that belongs to `run`.

Meshes are the seeded jittered boxes of `kutta_b200.harness` (hexes, or six
tets per hex, RCM order) and the structured boxes of
`kutta_b200.coupled_harness`; sizes are the ones that the benchmark, the tests
and the fixtures use, or ragged ones around them. A mesh depends on its size
alone; coefficients, right-hand sides and flow fields come from the seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from kutta_b200 import coupled_harness, harness, learn
from kutta_b200 import linalg as L

M_MATRIX = L.OperatorStructure.SymmetricMMatrix


def listed():
    return [
        # The drop-in AMG-PCG on a few thousand ragged hex cells: a small 2D-like
        # or test case, where a solve is launches and latency only. V(5,5).
        dict(name="pressure_hex_small", kind="pressure", mesh="hex", nx=19, ny=17, nz=15,
             sweeps=5, rel_tol=1e-5),
        # The reference's own linear-algebra benchmark at its largest: 128^3
        # 7-point Poisson, seeded forcing, default V(5,5) cycle, relative 1e-6.
        dict(name="pressure_poisson128", kind="pressure", mesh="poisson", nx=128, ny=128, nz=128,
             sweeps=5, rel_tol=1e-6),
        # The same solver with the SST caller's V(2,2) on 663,552 tets, whose
        # pairwise hierarchy stalls at a large coarsest level.
        dict(name="pressure_tet48", kind="pressure", mesh="tet", nx=48, ny=48, nz=48, sweeps=2,
             rel_tol=1e-5),
        # AMG-BiCGStab on the non-symmetric upwind transport twin, 1,572,864 tets.
        dict(name="transport_tet64", kind="transport", mesh="tet", nx=64, ny=64, nz=64, sweeps=5,
             rel_tol=1e-6),
        # The mixed-precision solve on about ten thousand tets, tight tolerance:
        # launches, small levels and the FP64 refinement.
        dict(name="mixed_tet_small", kind="mixed", mesh="tet", nx=13, ny=12, nz=11, field="cells",
             learned=0, rel_tol=1e-8),
        # The mixed solve on 64^3 hexes with a smooth log-normal diffusivity (the
        # learned stage's training configuration).
        dict(name="mixed_hex64", kind="mixed", mesh="hex", nx=64, ny=64, nz=64, field="smooth",
             learned=0, rel_tol=1e-6),
        # The benchmark's headline: 5,308,416 tets, mixed solve with the learned
        # stage as its warm start, to relative 1e-6.
        dict(name="mixed_tet96", kind="mixed", mesh="tet", nx=96, ny=96, nz=96, field="cells",
             learned=1, rel_tol=1e-6),
        # The Coupled block solve with the steady solver's control: a 960-cell
        # closed box (a reference cell and its gauge), 196,608 tets with hub
        # rows on the coarse levels, and 884,736 hexes.
        dict(name="coupled_hex_small", kind="coupled", mesh="hex", nx=12, ny=10, nz=8, closed=1),
        dict(name="coupled_tet32", kind="coupled", mesh="tet", nx=32, ny=32, nz=32, closed=0),
        dict(name="coupled_hex96", kind="coupled", mesh="hex", nx=96, ny=96, nz=96, closed=0),
        # One training gradient of the learned stage on its 64^3 systems: the
        # network forward and backward.
        dict(name="train_hex64", kind="train", nx=64, ny=64, nz=64),
        # The steps around the solve on 1,572,864 tets: pressure assembly fused
        # with the refresh of the mixed hierarchy, flux and velocity corrections.
        dict(name="outer_tet64", kind="outer", mesh="tet", nx=64, ny=64, nz=64),
    ]


def _sides(rng, low, high):
    """Three sides whose product is log-uniform in [low, high], up to a factor
    of 1.7 apart from one another and rarely round."""
    cells = math.exp(rng.uniform(math.log(low), math.log(high)))
    side = cells ** (1 / 3)
    a, b = rng.uniform(0.75, 1.3), rng.uniform(0.75, 1.3)
    nx, ny = max(3, round(side * a)), max(3, round(side * b))
    return dict(nx=nx, ny=ny, nz=max(3, int(cells / (nx * ny))))


def draw(rng):
    kind = rng.choice(["pressure", "pressure", "transport", "mixed", "mixed", "coupled", "coupled",
                       "train", "outer"])
    tet = rng.random() < 0.5
    case = dict(kind=kind)
    if kind == "pressure":
        mesh = rng.choice(["hex", "tet", "poisson"])
        top = {"hex": 700_000, "tet": 110_000, "poisson": 2_000_000}[mesh]
        case.update(mesh=mesh, sweeps=rng.choice([5, 2]),
                    rel_tol=1e-6 if mesh == "poisson" else 1e-5, **_sides(rng, 400, top))
    elif kind == "transport":
        case.update(mesh="tet" if tet else "hex", sweeps=5, rel_tol=1e-6,
                    **_sides(rng, 400, 260_000 if tet else 1_000_000))
    elif kind == "mixed":
        case.update(mesh="tet" if tet else "hex", field=rng.choice(["cells", "smooth"]),
                    learned=rng.choice([0, 1]), rel_tol=rng.choice([1e-6, 1e-8]),
                    **_sides(rng, 400, 260_000 if tet else 1_000_000))
    elif kind == "coupled":
        case.update(mesh="tet" if tet else "hex", closed=rng.choice([0, 0, 1]),
                    **_sides(rng, 300, 60_000 if tet else 800_000))
    elif kind == "train":
        case.update(**_sides(rng, 2_000, 262_144))
    else:
        case.update(mesh="tet" if tet else "hex", **_sides(rng, 400, 260_000 if tet else 1_000_000))
    return case


# ---- inputs ---------------------------------------------------------------------

@functools.lru_cache(maxsize=2)
def _mesh(mesh, nx, ny, nz, convection):
    """The system of a box, and what re-valuing it needs on the device."""
    if mesh == "poisson":
        s = harness.poisson(nx, ny, nz)
    else:
        s = harness.box_system(nx, ny, nz, tet=mesh == "tet", seed=1, convection=convection)
    cuda = {"row": torch.repeat_interleave(torch.arange(s.n, device="cuda"),
                                           torch.from_numpy(np.diff(s.row_ptr)).cuda()),
            "col": torch.from_numpy(s.col).cuda().long(),
            "diag": torch.from_numpy(s.diag).cuda().long()}
    if mesh != "poisson":
        cuda["geometry"] = torch.from_numpy(s.geometry).cuda()
        cuda["boundary"] = torch.from_numpy(s.boundary).cuda()
        cuda["centroid"] = torch.from_numpy(s.centroid).cuda()
        cuda["volume"] = torch.from_numpy(s.volume).cuda()
    return s, cuda


@functools.lru_cache(maxsize=2)
def _coupled_mesh(mesh, nx, ny, nz, closed):
    kinds = (0,) * 6 if closed else (1, 2, 0, 0, 3, 3)
    box = coupled_harness.box_tet if mesh == "tet" else coupled_harness.box_hex
    arrays = box(nx, ny, nz, patch_kinds=kinds)
    return arrays, L.CoupledMesh(arrays)


@functools.lru_cache(maxsize=1)
def _faces(mesh, nx, ny, nz):
    s, _ = _mesh(mesh, nx, ny, nz, 0.0)
    return harness.fv_faces(s.row_ptr, s.col, s.diag, seed=1)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _values(cuda, field, g):
    """Face coefficients 0.5 (D_P + D_N) |A_f| / |c_N - c_P| of a seeded
    diffusivity, as the M-matrix that the pressure assembly stores: float
    off-diagonals, each diagonal the upward-rounded sum of their magnitudes and
    its boundary term. D per cell log-uniform in [1e-3, 1], or a smooth
    log-normal field (sigma 1.5, correlation length 0.1)."""
    n = cuda["diag"].numel()
    if field == "smooth":
        wave = _randn(g, 3, 64) / 0.1
        shift = _rand(g, 64) * (2 * math.pi)
        total = torch.zeros(n, device="cuda", dtype=torch.float64)
        for q in range(64):
            total += torch.cos(cuda["centroid"] @ wave[:, q] + shift[q])
        d = torch.exp(1.5 * math.sqrt(2 / 64) * total)
    else:
        d = torch.exp(math.log(1e-3) * _rand(g, n))
    off = (0.5 * (d[cuda["row"]] + d[cuda["col"]]) * cuda["geometry"]).float().double()
    total = torch.zeros(n, device="cuda", dtype=torch.float64).index_add_(0, cuda["row"], off)
    total += cuda["boundary"]
    up = total.float()
    up = torch.where(up.double() < total, torch.nextafter(up, torch.full_like(up, math.inf)), up)
    val = -off
    val[cuda["diag"]] = up.double()
    return val


def _modes(cuda, g):
    """16 Fourier modes over the cell centroids and 10 % white noise."""
    wave = torch.randint(1, 5, (3, 16), generator=g, device="cuda").double() * (2 * math.pi)
    field = torch.sin(cuda["centroid"] @ wave + 2 * math.pi * _rand(g, 16)) @ _randn(g, 16)
    return field + 0.1 * field.square().mean().sqrt() * _randn(g, field.numel())


def _system(case, seed):
    """(host CSR with this seed's values, its right-hand side in float32)."""
    kind, mesh = case["kind"], case.get("mesh", "hex")
    s, cuda = _mesh(mesh, case["nx"], case["ny"], case["nz"],
                    1e-3 if kind == "transport" else 0.0)
    g = _generator(seed)
    if mesh == "poisson":
        val = s.val
        b = torch.randint(-1000, 1001, (s.n,), generator=g, device="cuda").float() / 1024
    else:
        field = "smooth" if kind == "train" else case.get("field", "cells")
        val = s.val if kind == "transport" else _values(cuda, field, g).cpu().numpy()
        b = _modes(cuda, g) if field == "smooth" else _randn(g, s.n)
        b = (b * cuda["volume"]).float()
    return L.CsrMatrixHost(s.n, s.row_ptr, s.col, s.diag, val), b


def prepare(case, seed):
    kind = case["kind"]
    if kind == "coupled":
        return _prepare_coupled(case, seed)
    host, b = _system(case, seed)
    a = L.upload(host)
    st = dict(case=case, a=a, b=b)
    if kind in ("pressure", "transport"):
        options = L.AmgOptions(pre_sweeps=case["sweeps"], post_sweeps=case["sweeps"])
        if kind == "pressure":
            options.structure = M_MATRIX
        st["solver"] = L.make_amg_solver(
            L.SolverKind.AmgPcg if kind == "pressure" else L.SolverKind.AmgBicgstab, host, options)
        st["x"] = torch.zeros_like(b)
        st["control"] = L.SolveControl(case["rel_tol"], 1e-30, 500)
    elif kind == "mixed":
        st["solver"] = L.make_mixed_solver(host)
        if case["learned"]:
            st["solver"].set_learned(learn.trained_stage(), L.LEARNED_WARM_START)
        st["x"] = torch.zeros_like(b, dtype=torch.float64)
        st["control"] = L.SolveControl(case["rel_tol"], 1e-30, 3000)
    elif kind == "train":
        st["stage"] = learn.trained_stage()
        st["stage"].bind(a)
        st["e"], st["t"] = _pair(case, a, seed)
    else:
        _prepare_outer(st, case, host, seed)
    return st


def _pair(case, a, seed):
    """(e, t) with A e = t: a smooth error with 10 % noise, as a cycle leaves."""
    _, cuda = _mesh("hex", case["nx"], case["ny"], case["nz"], 0.0)
    e = _modes(cuda, _generator(seed + 1_000_003)).float()
    t = torch.zeros(a.n_rows, device="cuda", dtype=torch.float64)
    t.index_add_(0, cuda["row"], a.val.double() * e.double()[cuda["col"]])
    return e, t.float()


def _prepare_outer(st, case, host, seed):
    c = _faces(case["mesh"], case["nx"], case["ny"], case["nz"])
    g = _generator(seed + 2_000_003)
    n = host.n_rows

    def on(x):
        return torch.from_numpy(np.ascontiguousarray(x)).cuda()

    coefficient = torch.exp(math.log(1e-3) * _rand(g, c.n_faces)).float()
    st["fv"] = L.FvPressure(on(c.offsets), on(c.faces), on(c.sign), on(c.adjacent), on(c.entry),
                            coefficient, _randn(g, c.n_faces).float(), -1)
    st["owner"], st["neighbour"], st["internal"] = on(c.owner), on(c.neighbour), c.internal
    st["rhs"] = torch.zeros(n, device="cuda")
    st["correction"] = _randn(g, n).float()
    st["cells"] = [(0.5 + _rand(g, n)).float() for _ in range(3)]
    st["gradient"] = [_randn(g, n).float() for _ in range(3)]
    st["fields"] = [torch.zeros(n, device="cuda") for _ in range(4)]
    st["solver"] = L.make_mixed_solver(host)


def _prepare_coupled(case, seed):
    arrays, mesh = _coupled_mesh(case["mesh"], case["nx"], case["ny"], case["nz"], case["closed"])
    reference = 0 if case["closed"] else -1
    fields = coupled_harness.flow_fields(arrays, seed, reference=reference)
    st = dict(case=case, solver=L.CoupledSolver(mesh, reference, L.CoupledOptions()),
              control=L.SolveControl(0.1, 1e-12, 20))
    st["fields"] = {k: torch.from_numpy(v).cuda() if isinstance(v, np.ndarray) else v
                    for k, v in fields.items()}
    st["rows"] = torch.from_numpy(arrays["pattern_row_ptr"]).cuda()
    st["diag"] = torch.from_numpy(arrays["pattern_diag"]).cuda()
    # The fields that the solves update, one relaxed step each: from zero here,
    # so that what comes back is the steps themselves.
    st["flow"] = [torch.zeros(mesh.n_cells, device="cuda") for _ in range(4)]
    return st


# ---- one pass -------------------------------------------------------------------

def run(st):
    kind = st["case"]["kind"]
    if kind == "coupled":
        f = st["fields"]
        for k, c in enumerate("uvw"):
            st["solver"].capture_diagonal(k, st["rows"], st["diag"], f["momentum_" + c],
                                          f["physical_" + c])
        st["solver"].solve(f, st["control"])
        st["solver"].update(*st["flow"], 0.7, 0.3)
        return dict(zip("uvwp", st["flow"]))
    if kind == "train":
        gradient, loss = st["stage"].gradient(st["t"], st["e"])
        return {"gradient": gradient, "loss": loss}
    if kind == "outer":
        st["solver"].assemble_refresh(st["a"], st["fv"], st["rhs"])
        L.fv_correct_flux(st["owner"], st["neighbour"], st["correction"], st["fv"].coefficient,
                          st["fv"].flux, st["internal"])
        L.fv_correct_velocity(*st["cells"], *st["gradient"], st["correction"], *st["fields"], 0.3)
        return {"values": st["a"].val, "rhs": st["rhs"], "flux": st["fv"].flux,
                **dict(zip("uvwp", st["fields"]))}
    st["solver"].refresh(st["a"])
    st["x"].zero_()
    st["solver"].solve(st["a"], st["x"], st["b"], st["control"])
    return {"x": st["x"]}


def _counts(case):
    """(cells, internal faces, boundary faces) of a case's box."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    boxes, sides = nx * ny * nz, nx * ny + ny * nz + nz * nx
    if case.get("mesh") != "tet":
        return boxes, 3 * boxes - sides, 2 * sides
    return 6 * boxes, 12 * boxes - 2 * sides, 4 * sides


def work(case):
    n, internal, boundary = _counts(case)
    nnz = n + 2 * internal
    csr = 8 * nnz + 8 * n
    kind = case["kind"]
    if kind == "coupled":
        # Mesh, geometry and least-squares arrays, momentum rows and residuals
        # in, the four fields read and written; one block row product.
        slots = 2 * internal + boundary
        faces = internal + boundary
        return {"bytes": 28 * slots + 44 * faces + 16 * nnz + 100 * n,
                "flops": 60.0 * internal + 40 * n}
    if kind == "train":
        # Two 32-wide layers of [H | W H] forward, their two products each
        # backward; the matrix, both vectors in and the gradient out.
        return {"bytes": csr + 8 * n, "flops": 3 * 2 * 2.0 * 64 * 32 * n}
    if kind == "outer":
        faces = int(1.1 * internal) + n // 3
        slots = 2 * int(1.1 * internal) + n // 3
        return {"bytes": 20 * slots + 20 * faces + 4 * nnz + 80 * n, "flops": 6.0 * slots + 20 * n}
    # Matrix and right-hand side in, solution out, and one product with A.
    return {"bytes": csr + (12 if kind == "mixed" else 8) * n, "flops": 2.0 * nnz}


def tolerance(case):
    """About four times what a right-hand side changed at random in its last
    float bit does to the result (pressure up to 2.1e-6, transport 7e-8, mixed
    1.2e-7, coupled 4.6e-6), with room in the pressure solves for a stop one
    update earlier or later, which moves x by up to its own error (3.6e-5 and
    8.1e-6 against 64 bits). The training gradient rounds its tile operands to
    BF16 (1.1e-3 against 64 bits); the outer steps are sums of a few floats."""
    return {"rel": {"pressure": 2e-5, "transport": 1e-6, "mixed": 1e-5, "coupled": 3e-5,
                    "train": 1e-3, "outer": 1e-6}[case["kind"]]}


# ---- the same in 64 bits ------------------------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind == "coupled":
        return None  # an iterate at relative 0.1: 64 bits have no such value
    host, b = _system(case, seed)
    n = host.n_rows
    val = torch.from_numpy(host.val).cuda()
    mesh, convection = case.get("mesh", "hex"), 1e-3 if kind == "transport" else 0.0
    _, cuda = _mesh(mesh, case["nx"], case["ny"], case["nz"], convection)
    if kind == "outer":
        return _exact_outer(case, host, cuda, seed)
    matrix = torch.sparse_csr_tensor(torch.from_numpy(host.row_ptr).cuda().long(), cuda["col"], val,
                                     (n, n))
    if kind == "train":
        a = L.CsrMatrix(n, host.nnz, None, None, None, val.float())
        e, t = _pair(case, a, seed)
        return _exact_gradient(cuda, matrix, val, t.double(), e.double())
    inverse = 1 / val[cuda["diag"]]
    solve = _bicgstab if kind == "transport" else _pcg
    return {"x": solve(matrix, inverse, b.double())}


def _pcg(a, inverse, b):
    """Jacobi-preconditioned conjugate gradients in FP64."""
    x, r = torch.zeros_like(b), b.clone()
    z = inverse * r
    p, rz, stop = z.clone(), r @ z, 1e-11 * b.norm()
    for k in range(20_000):
        q = a @ p
        alpha = rz / (p @ q)
        x += alpha * p
        r -= alpha * q
        if k % 20 == 0 and r.norm() <= stop:
            break
        z = inverse * r
        rz, old = r @ z, rz
        p = z + (rz / old) * p
    return x


def _bicgstab(a, inverse, b):
    """Jacobi-preconditioned BiCGStab in FP64."""
    x, r = torch.zeros_like(b), b.clone()
    shadow, p, v = r.clone(), torch.zeros_like(b), torch.zeros_like(b)
    rho = alpha = omega = torch.ones((), device=b.device, dtype=b.dtype)
    stop = 1e-12 * b.norm()
    for _ in range(1_000):
        rho, old = shadow @ r, rho
        p = r + (rho / old) * (alpha / omega) * (p - omega * v)
        y = inverse * p
        v = a @ y
        alpha = rho / (shadow @ v)
        s = r - alpha * v
        z = inverse * s
        t = a @ z
        omega = (t @ s) / (t @ t)
        x += alpha * y + omega * z
        r = s - omega * t
        if r.norm() <= stop:
            break
    return x


def _exact_gradient(cuda, matrix, val, t, e):
    """The energy loss 1 - (c.t)^2 / ((c.A c)(t.e)), c = G(t), of the
    three-layer network with the packaged weights, and its gradient."""
    n, width = t.numel(), 32
    w = torch.from_numpy(np.load(learn.WEIGHTS)).cuda().double().requires_grad_()
    scale = val[cuda["diag"]].rsqrt()
    edge = -val * scale[cuda["row"]] * scale[cuda["col"]]
    edge[cuda["diag"]] = 0
    graph = torch.sparse_csr_tensor(matrix.crow_indices(), cuda["col"], edge, (n, n))
    h = scale * t
    rho = h.square().mean().sqrt()
    h, at = (h / rho)[:, None], 0
    for inputs in (1, width, width):
        own = w[at:at + width * inputs].reshape(width, inputs)
        near = w[at + width * inputs:at + 2 * width * inputs].reshape(width, inputs)
        at += 2 * width * inputs
        bias = w[at:at + width]
        at += width
        # The graph is symmetric, so its product is its own adjoint.
        h = torch.relu(h @ own.T + _Symmetric.apply(graph, h) @ near.T + bias)
    c = rho * scale * (h @ w[at:at + width])
    loss = 1 - (c @ t).square() / ((c @ _Symmetric.apply(matrix, c[:, None])[:, 0]) * (t @ e))
    loss.backward()
    return {"gradient": w.grad, "loss": loss.detach()}


class _Symmetric(torch.autograd.Function):
    """Y = S X for a symmetric sparse S, with dX = S dY."""

    @staticmethod
    def forward(ctx, s, x):
        ctx.s = s
        return s @ x

    @staticmethod
    def backward(ctx, grad):
        return None, ctx.s @ grad


def _exact_outer(case, host, cuda, seed):
    c = _faces(case["mesh"], case["nx"], case["ny"], case["nz"])
    g = _generator(seed + 2_000_003)
    n = host.n_rows
    coefficient = torch.exp(math.log(1e-3) * _rand(g, c.n_faces)).float().double()
    flux = _randn(g, c.n_faces).float().double()
    correction = _randn(g, n).float().double()
    volume, inverse, diagonal = [(0.5 + _rand(g, n)).float().double() for _ in range(3)]
    gradient = [_randn(g, n).float().double() for _ in range(3)]
    cell = torch.from_numpy(np.repeat(np.arange(n), np.diff(c.offsets))).cuda()
    face = torch.from_numpy(c.faces).cuda().long()
    entry = torch.from_numpy(c.entry).cuda().long()
    sign = torch.from_numpy(c.sign).cuda().double()
    inner = torch.from_numpy(c.adjacent).cuda() >= 0
    values = torch.zeros(host.nnz, device="cuda", dtype=torch.float64)
    values.index_add_(0, entry[inner], -coefficient[face[inner]])
    total = torch.zeros(n, device="cuda", dtype=torch.float64)
    total.index_add_(0, cell, coefficient[face])
    values[cuda["diag"]] = total
    rhs = torch.zeros(n, device="cuda", dtype=torch.float64)
    rhs.index_add_(0, cell, -sign * flux[face])
    owner, near = torch.from_numpy(c.owner).cuda().long(), torch.from_numpy(c.neighbour).cuda().long()
    flux += coefficient * correction[owner]
    flux[:c.internal] -= coefficient[:c.internal] * correction[near]
    step = volume * inverse
    alpha = torch.minimum(torch.full_like(inverse, 0.3), 0.7 * diagonal * inverse)
    return {"values": values, "rhs": rhs, "flux": flux, "p": alpha * correction,
            **{k: -step * d for k, d in zip("uvw", gradient)}}
