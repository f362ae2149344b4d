"""Solves of both precisions on one operator, in the order in which the workspace that they
share grows after the mixed solver's first use of it: mixed, FP64 (a solve, or the timing of
its kernels), mixed. The third call repeats the first, and objects made in between keep
their contents."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOX = (1000.0, 1000.0, 600.0)


def make_op(orc, geo, dpn, shape):
    xyz, conn = orc.generate_cube(*shape, *BOX)
    mask, vals = orc.thermal_bc(xyz, BOX[2])
    dm = geo.DofManager(xyz.shape[0], dpn)
    idx = np.nonzero(np.repeat(mask, dpn))[0]
    dm.set_dirichlet(idx, np.repeat(vals, dpn)[idx] * (1.0 if dpn == 1 else 1e-3))
    mesh = geo.Mesh(xyz, conn)
    if dpn == 1:
        return geo.ThermalOperator(mesh, dm, np.full(conn.shape[0], 3.0))
    return geo.ElasticityOperator(mesh, dm, geo.IsotropicElasticity(1e11, 0.25), np.full(conn.shape[0], 1e11))


@pytest.mark.parametrize("between", ["solve", "timing"])
@pytest.mark.parametrize("halo", ["default", "atomics"])
@pytest.mark.parametrize("dpn,shape", [(1, (6, 6, 6)), (1, (13, 11, 9)), (3, (5, 4, 4))])
def test_mixed_fp64_mixed(orc, geo, monkeypatch, dpn, shape, halo, between):
    from geo_simulator_b200 import _native as N
    if halo == "atomics":
        monkeypatch.setenv("GEO_PATCH_HALO", "0")  # read when an operator is made
    tol = 1e-9
    solver = {p: geo.ConjugateGradient().with_tolerance(tol).with_max_iterations(20000).with_precision(p)
              for p in ("fp64", "mixed")}
    op = make_op(orc, geo, dpn, shape)
    n = op.n_dofs
    fb = op.lift_rhs(np.random.default_rng(3).standard_normal(n))
    first, st = op.solve(fb, solver["mixed"])
    assert st.converged and st.fp64_residual_updates >= 2
    if between == "solve":
        op.solve(fb, solver["fp64"])
    else:
        ms = (ctypes.c_double(), ctypes.c_double())
        assert N.lib().geo_op_time_pcg_kernels(op.h, fb.ctypes.data, N.PRECISION_FP64, 3, *map(ctypes.byref, ms)) == 0
    # matrices whose entries are as many as a vector of the workspace has, and another operator
    fill = np.random.default_rng(4).standard_normal(n)
    others = [geo.CsrMatrix.from_arrays(n, n, np.arange(n + 1), np.arange(n), fill * (i + 1)) for i in range(24)]
    op2 = make_op(orc, geo, dpn, shape)
    fb2 = op2.lift_rhs(np.random.default_rng(5).standard_normal(n))
    before = op2.solve(fb2, solver["mixed"])[0]
    third, st3 = op.solve(fb, solver["mixed"])
    after = op2.solve(fb2, solver["mixed"])[0]
    for i, A in enumerate(others):
        assert np.array_equal(A.to_host()[2], fill * (i + 1)), i
    # the true residual is the one the solver stopped on
    for o, b, xs in ((op, fb, (first, third)), (op2, fb2, (before, after))):
        for x in xs:
            assert np.linalg.norm(b - o.apply(x)) <= 2 * tol * np.linalg.norm(b)
    assert st3.converged
    if halo == "default":  # fixed-order sums: the same bits again
        assert np.array_equal(third, first) and np.array_equal(after, before)
