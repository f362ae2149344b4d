"""The PCG loop's launch forms: kernels started before the one before them has ended (up to
2.5 M dofs), and not (above). A solution's residual, formed by the operator apply, meets
the tolerance that the solver says it met."""
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
