"""The PCG loop's launch forms: kernels started before the one before them has ended (up to
2.5 M dofs), and not (above). A solution's residual, formed by the operator apply, meets
the tolerance that the solver says it met. And the iteration limit inside, at the end and
behind the end of a pass of the loop."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one patch; a last chunk of iterations that is cut short; 2.57 M dofs
CASES = [("thermal", (1, 1, 1)), ("thermal", (13, 3, 2)), ("elastic", (5, 4, 4)), ("elastic", (47, 47, 47))]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("physics,shape", CASES)
def test_residual_of_solution(orc, geo, physics, shape, precision):
    box = (1000.0, 1000.0, 600.0)
    xyz, conn = orc.generate_cube(*shape, *box)
    dpn = 1 if physics == "thermal" else 3
    mask, vals = orc.thermal_bc(xyz, box[2])
    dm = geo.DofManager(xyz.shape[0], dpn)
    idx = np.nonzero(np.repeat(mask, dpn))[0]
    dm.set_dirichlet(idx, np.repeat(vals, dpn)[idx] * (1.0 if dpn == 1 else 1e-3))
    mesh = geo.Mesh(xyz, conn)
    if dpn == 1:
        op = geo.ThermalOperator(mesh, dm, np.full(conn.shape[0], 3.0))
    else:
        op = geo.ElasticityOperator(mesh, dm, geo.IsotropicElasticity(1e11, 0.25), np.full(conn.shape[0], 1e11))
    f = np.random.default_rng(3).standard_normal(dpn * xyz.shape[0])
    fb = op.lift_rhs(f)
    tol = 1e-6
    solver = geo.ConjugateGradient().with_tolerance(tol).with_max_iterations(20000).with_precision(precision)
    x, st = op.solve(fb, solver)
    assert st.converged
    # the recursive residual of FP64 PCG leaves the true one by rounding, far below 1e-6
    assert np.linalg.norm(fb - op.apply(x)) <= 2 * tol * np.linalg.norm(fb)
    # and the same bits again: every sum has a fixed order
    x2, st2 = op.solve(fb, solver)
    assert st2.iterations == st.iterations and np.array_equal(x, x2)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("limit", [1, 15, 16, 17, 33])
def test_iteration_limit(orc, geo, limit, precision):
    box = (1000.0, 1000.0, 600.0)
    xyz, conn = orc.generate_cube(6, 6, 6, *box)
    mask, vals = orc.thermal_bc(xyz, box[2])
    dm = geo.DofManager(xyz.shape[0], 1)
    idx = np.nonzero(mask)[0]
    dm.set_dirichlet(idx, vals[idx])
    op = geo.ThermalOperator(geo.Mesh(xyz, conn), dm, np.full(conn.shape[0], 3.0))
    fb = op.lift_rhs(np.zeros(xyz.shape[0]))
    x, st = op.solve(fb, geo.ConjugateGradient().with_tolerance(1e-12).with_max_iterations(limit).with_precision(precision))
    assert st.iterations == limit and not st.converged
    # the solution left behind belongs to the last iteration: its residual is the one reported
    true = np.linalg.norm(fb - op.apply(x))
    bar = 1e-9 if precision == "fp64" else 1e-5  # rounding of the recursion; of the FP32 correction
    assert abs(true - st.residual_norm) <= bar * np.linalg.norm(fb)
