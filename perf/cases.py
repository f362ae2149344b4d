"""Performance cases: the calls that programs built on this package spend their time in.

A case names a call sequence (``kind``), a mesh (a box of nx x ny x nz hexes cut into
6 Tet10 each, straight, smoothly warped with straight edges, or curved), a physics and
the options of the call. ``prepare`` makes what a program has in hand before the call
(mesh, DOFs, coefficients, operator or matrix), ``run`` is one pass through the public
API, ``exact`` is the same result in plain torch FP64 on an independent lattice mesh.

Kinds
  forward    ``operator.forward(f, solver)``: lift the load, matrix-free PCG, u
  inversion  one step of a coefficient inversion: ``set_coefficients``, ``forward``,
             residual at the observed DOFs, ``vjp``
  apply      ``operator.apply(x, precision)``
  maxwell    one viscoelastic time step: ``BackwardEuler.step_operator`` and
             ``update_stresses_maxwell`` (host arrays, as the time loop keeps them)
  assemble   ``Assembler.assemble_*_stiffness_parallel`` and ``apply_dirichlet_bcs``
  krylov     ``ConjugateGradient`` / ``BiCGSTAB`` ``.solve(K_bc, f_bc)`` on the CSR
  direct     ``DirectSolver.solve(K_bc, f_bc)``
  pipeline   from host arrays to the solution: mesh, DOFs, operator, load, forward
"""
from __future__ import annotations

import math

import numpy as np
import torch

import geo_simulator_b200 as geo
from geo_simulator_b200 import _native

THERMAL_BOX = (1000.0, 1000.0, 600.0)
ELASTIC_BOX = (100e3, 100e3, 50e3)
YOUNG, POISSON, DENSITY, GRAVITY, VISCOSITY = 1e11, 0.25, 3300.0, 9.81, 1e19


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # The smallest thermal benchmark (6^3 hexes, 2,197 DOFs) in plain FP64: a call
        # whose time is launches and latency, as in unit checks and parameter sweeps.
        _case("thermal_6_fp64", "forward", "thermal", 6, 6, 6, tol=1e-10),
        # Plain FP64 matrix-free solve of the 64^3 cube with one uniform conductivity.
        _case("thermal_64_fp64", "forward", "thermal", 64, 64, 64, tol=1e-12, sigma=0.0),
        # The largest configuration: 17M DOFs, log-normal conductivity, mixed precision,
        # converged far enough that mixed and FP64 solutions agree.
        _case("thermal_128_mixed", "forward", "thermal", 128, 128, 128, tol=1e-13, precision="mixed", sigma=0.5),
        # One step of the thermal inversion: new coefficients, forward, adjoint gradient,
        # converged as far as a gradient check asks.
        _case("inversion_48x48x32_mixed", "inversion", "thermal", 48, 48, 32, tol=2e-14, precision="mixed",
              sigma=0.3),
        # Half-space under gravity, 1.4M DOFs, heterogeneous stiffness, mixed precision.
        _case("elastic_48x48x24_mixed", "forward", "elastic", 48, 48, 24, tol=1e-10, precision="mixed", sigma=0.3),
        # One viscoelastic time step in FP64 on a ragged box.
        _case("maxwell_27x22x13_fp64", "maxwell", "elastic", 27, 22, 13, tol=1e-10, sigma=0.0),
        # The assembled drop-in path: stiffness CSR and Dirichlet elimination at 64^3.
        _case("assemble_thermal_64", "assemble", "thermal", 64, 64, 64, sigma=0.5),
        # The same for 3-DOF elasticity.
        _case("assemble_elastic_24x24x12", "assemble", "elastic", 24, 24, 12, sigma=0.3),
        # The CG drop-in on an assembled matrix with odd sizes.
        _case("csr_cg_45x37x29", "krylov", "thermal", 45, 37, 29, tol=1e-12, sigma=0.5, solver="cg"),
        # The direct solver on a small problem (3,757 unknowns), its usual range.
        _case("direct_8x8x6", "direct", "thermal", 8, 8, 6, sigma=0.5),
        # One application of the operator on a curved mesh with odd sizes, as an outer
        # method that brings its own iteration calls it.
        _case("apply_curved_45x37x29_fp64", "apply", "thermal", 45, 37, 29, sigma=0.5, shape="curved"),
        # A program that solves once: host arrays in, solution out.
        _case("pipeline_48x40x32_mixed", "pipeline", "thermal", 48, 40, 32, tol=1e-12, precision="mixed", sigma=0.5),
    ]


def _case(name, kind, phys, nx, ny, nz, tol=0.0, precision="fp64", sigma=0.0, shape="cube", solver=""):
    c = {"kind": kind, "phys": phys, "nx": nx, "ny": ny, "nz": nz, "tol": tol, "precision": precision,
         "sigma": sigma, "shape": shape, "solver": solver}
    return dict(c, name=name) if name else c


# hexes per axis, smallest and largest, by kind and physics
_RANGE = {
    ("forward", "thermal"): (4, 104), ("forward", "elastic"): (3, 40),
    ("inversion", "thermal"): (4, 48), ("inversion", "elastic"): (3, 32),
    ("apply", "thermal"): (4, 112), ("apply", "elastic"): (3, 48),
    ("maxwell", "elastic"): (3, 32),
    ("assemble", "thermal"): (4, 64), ("assemble", "elastic"): (3, 28),
    ("krylov", "thermal"): (4, 56), ("krylov", "elastic"): (3, 20),
    ("direct", "thermal"): (3, 8), ("direct", "elastic"): (2, 5),
    ("pipeline", "thermal"): (4, 72), ("pipeline", "elastic"): (3, 32),
}


def draw(rng):
    kind, phys = rng.choice(sorted(_RANGE))
    lo, hi = _RANGE[(kind, phys)]
    base = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    n = [min(hi, max(lo, round(base * math.exp(rng.uniform(-0.25, 0.25))))) for _ in range(3)]
    solves = kind in ("forward", "inversion", "maxwell", "krylov", "pipeline")
    tol = rng.choice([1e-12, 1e-13] if phys == "thermal" else [1e-10, 1e-11]) if solves else 0.0
    if kind == "inversion":
        tol = 2e-14 if phys == "thermal" else 1e-11
    precision = rng.choice(["fp64", "mixed"]) if kind in ("forward", "inversion", "apply", "maxwell", "pipeline") else "fp64"
    sigma = 0.0 if kind == "maxwell" else rng.choice([0.0, 0.3, 0.5])
    shape = "cube" if kind == "pipeline" else rng.choice(["cube", "cube", "warped", "curved"])
    solver = rng.choice(["cg", "cg", "bicgstab"]) if kind == "krylov" else ""
    return _case("", kind, phys, *n, tol=tol, precision=precision, sigma=sigma, shape=shape, solver=solver)


def _counts(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return 6 * nx * ny * nz, (2 * nx + 1) * (2 * ny + 1) * (2 * nz + 1)


def work(case):
    """Bytes and operations of one pass that no form of the path avoids. An iteration of
    PCG reads the element data (connectivity, coefficient) and coordinates or the matrix
    once and streams its vectors; its count is estimated from the mesh and tolerance."""
    E, N = _counts(case)
    dpn = 1 if case["phys"] == "thermal" else 3
    n, kind = dpn * N, case["kind"]
    s = 4 if case["precision"] == "mixed" else 8
    apply_flops = E * (186 if dpn == 1 else 1092)
    apply_bytes = E * (40 + s) + N * 3 * s + 2 * n * s
    nnz = 28 * N * dpn * dpn
    iters = 0.43 * max(case["nx"], case["ny"], case["nz"]) * math.log(2.0 / case["tol"]) + 10 if case["tol"] else 0.0
    solve = {"bytes": iters * (apply_bytes + 6 * n * s), "flops": iters * (apply_flops + 12 * n)}
    if kind in ("forward", "maxwell", "pipeline"):
        return {"bytes": solve["bytes"] + E * 48 + 4 * n * 8, "flops": solve["flops"] + apply_flops}
    if kind == "inversion":
        return {"bytes": 2 * solve["bytes"] + 2 * E * 48 + 6 * n * 8, "flops": 2 * solve["flops"] + 3 * apply_flops}
    if kind == "apply":
        return {"bytes": apply_bytes, "flops": apply_flops}
    if kind == "assemble":
        return {"bytes": E * 48 + N * 24 + 3 * nnz * 12, "flops": E * (2000 if dpn == 1 else 15000)}
    if kind == "krylov":
        passes = 2 if case["solver"] == "bicgstab" else 1
        return {"bytes": iters * (passes * nnz * 12 + 10 * n * 8), "flops": iters * (passes * 2 * nnz + 12 * n)}
    return {"bytes": nnz * 12 + 3 * n * 8, "flops": 2.0 / 3.0 * n ** 3}  # direct


# ------------------------------------------------------------------ inputs, shared by both sides
def _box(case):
    return THERMAL_BOX if case["phys"] == "thermal" else ELASTIC_BOX


def _displace(case, xyz):
    """Smooth displacement that vanishes on the box surface (torch or numpy [n, 3])."""
    lib = torch if isinstance(xyz, torch.Tensor) else np
    r = np.random.RandomState(case["nx"] * 10007 + case["ny"] * 101 + case["nz"])
    amp, freq = 0.02 * r.uniform(0.5, 1.0, 3), r.randint(1, 3, 3)
    box = _box(case)
    bump = 1.0
    for c in range(3):
        bump = bump * lib.sin(math.pi * xyz[:, c] / box[c])
    out = [xyz[:, c] + amp[c] * box[c] * bump * lib.cos(math.pi * float(freq[c]) * xyz[:, (c + 1) % 3] / box[(c + 1) % 3])
           for c in range(3)]
    return lib.stack(out, -1)


_EDGES = ((0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3))


def _shape(case, xyz, conn):
    """Coordinates of the case's shape from those of the straight box."""
    if case["shape"] == "cube":
        return xyz
    moved = _displace(case, xyz)
    if case["shape"] == "curved":
        return moved
    for k, (a, b) in enumerate(_EDGES):  # warped: vertices moved, midpoints on the straight edges
        moved[conn[:, 4 + k]] = (moved[conn[:, a]] + moved[conn[:, b]]) / 2.0
    return moved


def _inputs(case, seed):
    """Seeded coefficients and loads; the same on both sides."""
    E, N = _counts(case)
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    mean = math.log(3.0 if case["phys"] == "thermal" else YOUNG)
    coef = torch.exp(mean + case["sigma"] * torch.randn(E, generator=g, device="cuda", dtype=torch.float64))
    r = np.random.RandomState(seed % (1 << 31))
    load = r.uniform(0.5, 1.5)
    return coef, load, g, r


def _constraints(case, xyz):
    """Dirichlet DOFs and values (numpy): fixed temperatures at bottom and top, or a fixed
    base with roller sides."""
    box = _box(case)
    x, y, z = (xyz[:, c] for c in range(3))
    if case["phys"] == "thermal":
        bottom, top = np.nonzero(np.abs(z) < 1.0)[0], np.nonzero(np.abs(z - box[2]) < 1.0)[0]
        return np.concatenate([bottom, top]), np.concatenate([np.full(bottom.size, 1280.0), np.zeros(top.size)])
    base = np.nonzero(np.abs(z) < 1.0)[0]
    sx = np.nonzero((np.abs(x) < 1.0) | (np.abs(x - box[0]) < 1.0))[0]
    sy = np.nonzero((np.abs(y) < 1.0) | (np.abs(y - box[1]) < 1.0))[0]
    idx = np.unique(np.concatenate([3 * base, 3 * base + 1, 3 * base + 2, 3 * sx, 3 * sy + 1]))
    return idx, np.zeros(idx.size)


def _observed(case, xyz, r):
    """1000 observed temperatures or 500 vertical surface displacements, and their data."""
    z, box = xyz[:, 2], _box(case)
    if case["phys"] == "thermal":
        free = np.nonzero((np.abs(z) >= 1.0) & (np.abs(z - box[2]) >= 1.0))[0]
        at = np.sort(r.choice(free, min(1000, free.size), replace=False))
        return at, 1280.0 * (1.0 - z[at] / box[2]) + r.normal(0.0, 5.0, at.size)
    top = np.nonzero(np.abs(z - box[2]) < 1.0)[0]
    at = np.sort(r.choice(top, min(500, top.size), replace=False))
    return 3 * at + 2, r.normal(-400.0, 40.0, at.size)


# ------------------------------------------------------------------ prepare and run
class _State:
    pass


def _mesh(case):
    args = (case["nx"], case["ny"], case["nz"], *_box(case))
    if case["shape"] == "cube":
        return geo.ImprovedMeshGenerator.generate_cube_device(*args)
    m = geo.ImprovedMeshGenerator.generate_cube(*args)
    return geo.Mesh(_shape(case, m.nodes, m.elements), m.elements)


def _solver(case):
    if case["solver"] == "bicgstab":
        return geo.BiCGSTAB().with_tolerance(case["tol"]).with_max_iterations(50000)
    s = geo.ConjugateGradient().with_tolerance(case["tol"]).with_max_iterations(50000)
    return s.with_precision(case["precision"])


def _dofs(case, nodes):
    dm = geo.DofManager(nodes.shape[0], 1 if case["phys"] == "thermal" else 3)
    dm.set_dirichlet(*_constraints(case, nodes))
    return dm


def _load(case, mesh, dm, load):
    if case["phys"] == "thermal":
        return geo.Assembler.assemble_thermal_load(mesh, dm, 1e-6 * load)
    return geo.Assembler.assemble_gravity_load(mesh, dm, DENSITY, [0.0, 0.0, -GRAVITY * load])


def _operator(case, mesh, dm, coef):
    if case["phys"] == "thermal":
        return geo.ThermalOperator(mesh, dm, coef)
    return geo.ElasticityOperator(mesh, dm, geo.IsotropicElasticity(YOUNG, POISSON), coef)


def _assemble(case, mesh, dm, coef):
    if case["phys"] == "thermal":
        return geo.Assembler.assemble_thermal_stiffness_parallel(mesh, dm, coef)
    return geo.Assembler.assemble_elasticity_stiffness_parallel(mesh, dm, geo.IsotropicElasticity(YOUNG, POISSON), coef)


def prepare(case, seed):
    s = _State()
    s.case, kind = case, case["kind"]
    s.coef, load, g, r = _inputs(case, seed)
    torch.cuda.synchronize()
    # torch work of a pass is queued on the library's stream, in order with its calls
    s.stream = torch.cuda.ExternalStream(geo.Context.default().stream_handle())
    if kind == "pipeline":
        m = geo.ImprovedMeshGenerator.generate_cube(case["nx"], case["ny"], case["nz"], *_box(case))
        s.nodes, s.elements, s.coef, s.load = m.nodes, m.elements, s.coef.cpu().numpy(), load
        s.constraints, s.solver = _constraints(case, s.nodes), _solver(case)
        return s
    s.mesh = _mesh(case)
    s.dm = _dofs(case, s.mesh.nodes)
    n = s.dm.total_dofs()
    f = _load(case, s.mesh, s.dm, load)
    if kind in ("forward", "inversion"):
        s.f, s.solver = torch.from_numpy(f).cuda(), _solver(case)
        s.op = _operator(case, s.mesh, s.dm, s.coef)
        if kind == "inversion":
            at, data = _observed(case, s.mesh.nodes, r)
            s.at, s.data = torch.from_numpy(at).cuda(), torch.from_numpy(data).cuda()
    elif kind == "apply":
        s.x = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
        s.op = _operator(case, s.mesh, s.dm, s.coef)
    elif kind == "maxwell":
        s.material = geo.MaxwellViscoelasticity.new(YOUNG, POISSON, VISCOSITY)
        s.dt = 0.1 * s.material.relaxation_time()
        s.f, s.solver = f, _solver(case)
        s.mesh.stress_history = geo.StressHistory(s.mesh.num_elements())
        s.mesh.stress_history.update_all(r.normal(0.0, 1e6, (s.mesh.num_elements(), 6)))
        s.u = r.normal(0.0, 10.0, n)
        s.op = geo.ElasticityOperator(s.mesh, s.dm, geo.IsotropicElasticity(YOUNG, POISSON))
        s.be = geo.BackwardEuler.new(n, s.dt)
    elif kind == "assemble":
        s.f = f
    else:
        s.K, fb = geo.Assembler.apply_dirichlet_bcs(_assemble(case, s.mesh, s.dm, s.coef), f, s.dm)
        s.f = torch.from_numpy(fb).cuda()
        s.solver = geo.DirectSolver() if kind == "direct" else _solver(case)
    torch.cuda.synchronize()
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    with torch.cuda.stream(s.stream):
        if kind == "forward":
            return s.op.forward(s.f, s.solver)[0]
        if kind == "inversion":
            s.op.set_coefficients(s.coef)
            u, _ = s.op.forward(s.f, s.solver)
            dJ = torch.zeros_like(u)
            dJ[s.at] = u[s.at] - s.data
            return {"u": u, "gradient": s.op.vjp(dJ, u=u, solver=s.solver)[0]}
        if kind == "apply":
            return s.op.apply(s.x, case["precision"])
        if kind == "maxwell":
            u, _ = s.be.step_operator(s.op, s.mesh, s.f, s.solver)
            return {"u": u, "stress": geo.update_stresses_maxwell(s.mesh, s.dm, s.material, s.u, u, s.dt)}
        if kind == "assemble":
            K, fb = geo.Assembler.apply_dirichlet_bcs(_assemble(case, s.mesh, s.dm, s.coef), s.f, s.dm)
            # the matrix stays on the device: its arrays as torch tensors there
            indptr = torch.empty(K.rows() + 1, dtype=torch.int64, device="cuda")
            indices = torch.empty(K.nnz(), dtype=torch.int32, device="cuda")
            data = torch.empty(K.nnz(), dtype=torch.float64, device="cuda")
            K.ctx.check(_native.lib().geo_csr_copy(K.h, indptr.data_ptr(), indices.data_ptr(), data.data_ptr()))
            return {"indptr": indptr, "indices": indices, "data": data, "f": fb}
        if kind == "pipeline":
            mesh = geo.Mesh(s.nodes, s.elements)
            dm = geo.DofManager(mesh.num_nodes(), 1 if case["phys"] == "thermal" else 3)
            dm.set_dirichlet(*s.constraints)
            op = _operator(case, mesh, dm, s.coef)
            return op.forward(_load(case, mesh, dm, s.load), s.solver)[0]
        return s.solver.solve(s.K, s.f)[0]  # krylov, direct


# ------------------------------------------------------------------ exact, in plain torch
_QA, _QB, _QW = 0.5854101966249685, 0.1381966011250105, 1.0 / 24.0


def _lattice_mesh(case):
    """Nodes [N, 3] and elements [E, 10] of the box, numbered as the generator does:
    vertices, then edge midpoints in the order in which the elements first meet them."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    box = _box(case)
    dev = "cuda"
    ar = lambda n: torch.arange(n, device=dev)
    h = torch.tensor([box[0] / nx, box[1] / ny, box[2] / nz], dtype=torch.float64, device=dev)
    # vertices, x fastest
    vz, vy, vx = torch.meshgrid(ar(nz + 1), ar(ny + 1), ar(nx + 1), indexing="ij")
    vert = torch.stack([vx.reshape(-1), vy.reshape(-1), vz.reshape(-1)], -1)
    hz, hy, hx = torch.meshgrid(ar(nz), ar(ny), ar(nx), indexing="ij")
    base = torch.stack([hx.reshape(-1), hy.reshape(-1), hz.reshape(-1)], -1)  # [H, 3]
    corner = {c: torch.tensor([int(b) for b in c], device=dev) for c in
              ("000", "100", "010", "110", "001", "101", "011", "111")}
    tets = (("000", "100", "110", "111"), ("000", "100", "111", "101"), ("000", "010", "110", "111"),
            ("000", "010", "111", "011"), ("000", "001", "111", "101"), ("000", "001", "111", "011"))
    rows = []
    for t in tets:  # orient: swap the last two vertices where the volume is negative
        o = torch.stack([corner[c] for c in t]).double() * h
        neg = torch.linalg.det(o[1:] - o[0]) < 0
        rows.append(torch.stack([corner[c] for c in ((t[0], t[1], t[3], t[2]) if neg else t)]))
    corners = torch.stack(rows)  # [6, 4, 3]
    v4 = (base[:, None, None, :] + corners[None]).reshape(-1, 4, 3)  # [E, 4, 3] vertex lattice indices
    vid = v4[..., 0] + (nx + 1) * (v4[..., 1] + (ny + 1) * v4[..., 2])
    mids = torch.stack([v4[:, a] + v4[:, b] for a, b in _EDGES], 1)  # doubled-lattice indices
    lid = (mids[..., 0] + (2 * nx + 1) * (mids[..., 1] + (2 * ny + 1) * mids[..., 2])).reshape(-1)
    n_lat = (2 * nx + 1) * (2 * ny + 1) * (2 * nz + 1)
    never = torch.iinfo(torch.int64).max
    first = torch.full((n_lat,), never, device=dev).scatter_reduce_(0, lid, ar(lid.numel()), "amin")
    met = torch.nonzero(first != never).reshape(-1)
    met = met[torch.argsort(first[met])]
    number = torch.empty(n_lat, dtype=torch.int64, device=dev)
    number[met] = vert.shape[0] + ar(met.numel())
    conn = torch.cat([vid, number[lid].reshape(-1, 6)], 1)
    xyz = torch.empty((vert.shape[0] + met.numel(), 3), dtype=torch.float64, device=dev)
    xyz[: vert.shape[0]] = vert.double() * h
    for k, (a, b) in enumerate(_EDGES):
        xyz[conn[:, 4 + k]] = (xyz[conn[:, a]] + xyz[conn[:, b]]) / 2.0
    return _shape(case, xyz, conn), conn


def _quadrature():
    """Shape functions [4, 10] and reference gradients [4, 10, 3] at the 4 points."""
    N, G = torch.zeros(4, 10, dtype=torch.float64), torch.zeros(4, 10, 3, dtype=torch.float64)
    for q in range(4):
        L = [_QA if m == q else _QB for m in range(4)]
        for i in range(10):
            d = [0.0] * 4
            if i < 4:
                N[q, i] = L[i] * (2.0 * L[i] - 1.0)
                d[i] = 4.0 * L[i] - 1.0
            else:
                a, b = _EDGES[i - 4]
                N[q, i] = 4.0 * L[a] * L[b]
                d[a], d[b] = 4.0 * L[b], 4.0 * L[a]
            G[q, i] = torch.tensor([d[1] - d[0], d[2] - d[0], d[3] - d[0]], dtype=torch.float64)
    return N.cuda(), G.cuda()


def _geometry(X):
    """Cartesian gradients [4, e, 10, 3] and weights [4, e] of elements with nodes X [e, 10, 3]."""
    _, G = _quadrature()
    grads, weights = [], []
    for q in range(4):
        J = torch.einsum("eir,ic->erc", X, G[q])
        weights.append(_QW * torch.linalg.det(J).abs())
        grads.append(torch.einsum("ic,eca->eia", G[q], torch.linalg.inv(J)))
    return torch.stack(grads), torch.stack(weights)


def _element_matrices(case, xyz, conn, coef):
    dpn = 1 if case["phys"] == "thermal" else 3
    K = torch.empty((conn.shape[0], 10 * dpn, 10 * dpn), dtype=torch.float64, device="cuda")
    step = 1 << 18 if dpn == 1 else 1 << 15
    for e in range(0, conn.shape[0], step):
        g, w = _geometry(xyz[conn[e:e + step]])
        w = w * coef[e:e + step]
        if dpn == 1:
            K[e:e + step] = torch.einsum("qe,qeia,qeja->eij", w, g, g)
            continue
        lam = POISSON / ((1.0 + POISSON) * (1.0 - 2.0 * POISSON))
        mu = 0.5 / (1.0 + POISSON)
        out = torch.zeros((g.shape[1], 10, 3, 10, 3), dtype=torch.float64, device="cuda")
        for q in range(4):
            gw = w[q][:, None, None] * g[q]
            o = torch.einsum("eia,ejb->eiajb", gw, g[q])
            out += lam * o + mu * o.permute(0, 1, 4, 3, 2)
            dd = mu * torch.einsum("eia,eja->eij", gw, g[q])
            for a in range(3):
                out[:, :, a, :, a] += dd
        K[e:e + step] = out.reshape(-1, 30, 30)
    return K


class _System:
    """Matrix-free K in plain torch, its constraints and the load of a case."""

    def __init__(self, case, seed):
        self.case = case
        self.coef, self.load, self.g, self.r = _inputs(case, seed)
        if case["kind"] == "maxwell":
            self.coef = torch.full_like(self.coef, YOUNG)
        self.xyz, self.conn = _lattice_mesh(case)
        self.dpn = 1 if case["phys"] == "thermal" else 3
        self.n = self.dpn * self.xyz.shape[0]
        self.K = _element_matrices(case, self.xyz, self.conn, self.coef)
        self.dofs = (self.dpn * self.conn[:, :, None] + torch.arange(self.dpn, device="cuda")).reshape(self.conn.shape[0], -1)
        idx, vals = _constraints(case, self.xyz.cpu().numpy())
        self.fixed = torch.zeros(self.n, dtype=torch.bool, device="cuda")
        self.values = torch.zeros(self.n, dtype=torch.float64, device="cuda")
        self.fixed[torch.from_numpy(idx).cuda()] = True
        self.values[torch.from_numpy(idx).cuda()] = torch.from_numpy(vals).cuda()
        diag = self.scatter(torch.diagonal(self.K, dim1=1, dim2=2))
        self.char = max(1.0, float(diag.abs().max()))
        self.diag = torch.where(self.fixed, torch.full_like(diag, self.char), diag)

    def scatter(self, ve):
        return torch.zeros(self.n, dtype=torch.float64, device="cuda").index_add_(0, self.dofs.reshape(-1), ve.reshape(-1))

    def times(self, x):  # K x
        return self.scatter(torch.bmm(self.K, x[self.dofs].unsqueeze(-1)))

    def bc_times(self, x):  # K_bc x
        return torch.where(self.fixed, self.char * x, self.times(torch.where(self.fixed, torch.zeros_like(x), x)))

    def body_load(self):
        N, _ = _quadrature()
        f = torch.empty((self.conn.shape[0], 10, self.dpn), dtype=torch.float64, device="cuda")
        step = 1 << 18
        for e in range(0, self.conn.shape[0], step):
            _, w = _geometry(self.xyz[self.conn[e:e + step]])
            m = torch.einsum("qe,qi->ei", w, N)
            if self.dpn == 1:
                f[e:e + step, :, 0] = 1e-6 * self.load * m
            else:
                f[e:e + step] = 0.0
                f[e:e + step, :, 2] = -DENSITY * GRAVITY * self.load * m
        return self.scatter(f)

    def lift(self, f):  # f_bc
        return torch.where(self.fixed, self.char * self.values, f - self.times(torch.where(self.fixed, self.values, torch.zeros_like(f))))

    def solve(self, b):
        x = torch.zeros_like(b)
        r, z = b.clone(), b / self.diag
        p, rz = z.clone(), torch.dot(b, z)
        stop = 1e-15 * float(torch.linalg.norm(b))
        for i in range(20000):
            q = self.bc_times(p)
            a = rz / torch.dot(p, q)
            x.add_(a * p)
            r.sub_(a * q)
            z = r / self.diag
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
            if i % 16 == 15 and float(torch.linalg.norm(r)) <= stop:
                break
        return x

    def csr(self):
        """(indptr, indices, data) of K with one entry for every coupled pair of nodes."""
        nd = self.dofs.shape[1]
        key = (self.dofs[:, :, None] * self.n + self.dofs[:, None, :]).reshape(-1)
        pairs, at = torch.unique(key, return_inverse=True)
        data = torch.zeros(pairs.numel(), dtype=torch.float64, device="cuda").index_add_(0, at, self.K.reshape(-1))
        assert nd * nd * self.dofs.shape[0] == at.numel()
        return pairs // self.n, pairs % self.n, data


def _stress_update(s, dt, stress, u_n, u_next):
    """sigma_(n+1) of the Maxwell body: mean strain increment, elastic predictor, relaxation."""
    out = torch.empty_like(stress)
    G = YOUNG / (2.0 * (1.0 + POISSON))
    lam = YOUNG / (3.0 * (1.0 - 2.0 * POISSON)) - 2.0 * G / 3.0
    factor = 1.0 / (1.0 + dt * G / VISCOSITY)
    step = 1 << 17
    for e in range(0, s.conn.shape[0], step):
        g, _ = _geometry(s.xyz[s.conn[e:e + step]])
        du = (u_next - u_n)[s.dofs[e:e + step]].reshape(-1, 10, 3)
        F = torch.einsum("eic,qeib->ecb", du, g) / 4.0
        de = torch.stack([F[:, 0, 0], F[:, 1, 1], F[:, 2, 2], F[:, 0, 1] + F[:, 1, 0], F[:, 1, 2] + F[:, 2, 1],
                          F[:, 0, 2] + F[:, 2, 0]], -1)
        t = stress[e:e + step].clone()
        t[:, :3] += lam * de[:, :3].sum(1, keepdim=True) + 2.0 * G * de[:, :3]
        t[:, 3:] += G * de[:, 3:]
        p = t[:, :3].mean(1, keepdim=True)
        t[:, :3] = (t[:, :3] - p) * factor + p
        t[:, 3:] *= factor
        out[e:e + step] = t
    return out


def exact(case, seed):
    E, _ = _counts(case)
    kind = case["kind"]
    if E * (1 if case["phys"] == "thermal" else 9) > 8_000_000:
        return None  # over 20 seconds of plain torch
    s = _System(case, seed)
    if kind == "apply":
        x = torch.randn(s.n, generator=s.g, device="cuda", dtype=torch.float64)
        return s.bc_times(x)
    if kind == "maxwell":
        dt = 0.1 * VISCOSITY * 2.0 * (1.0 + POISSON) / YOUNG
        stress = torch.from_numpy(s.r.normal(0.0, 1e6, (s.conn.shape[0], 6))).cuda()
        u_n = torch.from_numpy(s.r.normal(0.0, 10.0, s.n)).cuda()
        fe = torch.empty((s.conn.shape[0], 10, 3), dtype=torch.float64, device="cuda")
        step = 1 << 17
        for e in range(0, s.conn.shape[0], step):
            g, w = _geometry(s.xyz[s.conn[e:e + step]])
            v = stress[e:e + step]
            S = torch.stack([v[:, [0, 3, 5]], v[:, [3, 1, 4]], v[:, [5, 4, 2]]], 1)
            fe[e:e + step] = -torch.einsum("qe,qeib,ecb->eic", w, g, S)
        u = s.solve(s.lift(s.body_load() + s.scatter(fe)))
        return {"u": u, "stress": _stress_update(s, dt, stress, u_n, u)}
    f = s.lift(s.body_load())
    if kind == "assemble":
        rows, cols, data = s.csr()
        keep = torch.where(s.fixed[rows], rows == cols, ~s.fixed[cols])
        rows, cols, data = rows[keep], cols[keep], data[keep]
        data = torch.where(s.fixed[rows], torch.full_like(data, s.char), data)
        indptr = torch.zeros(s.n + 1, dtype=torch.int64, device="cuda")
        indptr[1:] = torch.bincount(rows, minlength=s.n).cumsum(0)
        return {"indptr": indptr, "indices": cols.int(), "data": data, "f": f}
    if kind == "direct":
        rows, cols, data = s.csr()
        A = torch.zeros((s.n, s.n), dtype=torch.float64, device="cuda")
        A[rows, cols] = data
        A[s.fixed] = 0.0
        A[:, s.fixed] = 0.0
        A += torch.diag(torch.where(s.fixed, torch.full_like(f, s.char), torch.zeros_like(f)))
        return torch.linalg.solve(A, f)
    u = s.solve(f)
    if kind != "inversion":
        return u
    at, obs = _observed(case, s.xyz.cpu().numpy(), s.r)
    dJ = torch.zeros_like(u)
    dJ[torch.from_numpy(at).cuda()] = u[torch.from_numpy(at).cuda()] - torch.from_numpy(obs).cuda()
    dJ[s.fixed] = 0.0
    adj = s.solve(dJ)
    ke_u = torch.bmm(s.K, u[s.dofs].unsqueeze(-1)).squeeze(-1)
    return {"u": u, "gradient": -(adj[s.dofs] * ke_u).sum(1)}
