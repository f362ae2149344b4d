"""The patch kernel's aligned node groups at the sizes where they can go wrong: one
patch without foreign nodes, a patch of exactly 384 elements, a short last patch, node
counts that leave every remainder in the own ranges; straight and curved elements, one
and three DOFs per node. And two operators of different sizes alive at once: the shared
memory a kernel may take is the kernel's, not the operator's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (2, 1, 1), (4, 4, 4), (5, 4, 4), (13, 3, 2), (9, 8, 7)]


def curve(xyz, conn, box, shape):
    nv = np.unique(conn[:, :4]).size
    rng = np.random.default_rng(sum(shape))
    out = xyz.copy()
    out[nv:] += rng.uniform(-0.03, 0.03, (xyz.shape[0] - nv, 3)) * np.array(box) / np.array(shape)
    return out


@pytest.mark.parametrize("curved", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_apply_against_oracle(orc, geo, shape, curved):
    box = (1000.0, 1000.0, 600.0)
    xyz, conn = orc.generate_cube(*shape, *box)
    if curved:
        xyz = curve(xyz, conn, box, shape)
    mask, vals = orc.thermal_bc(xyz, box[2])
    rng = np.random.default_rng(7)
    k_e = np.exp(np.log(3.0) + 0.5 * rng.standard_normal(conn.shape[0]))
    E_e = np.exp(np.log(1e11) + 0.3 * rng.standard_normal(conn.shape[0]))
    mesh = geo.Mesh(xyz, conn)
    for dpn in (1, 3):
        m = np.repeat(mask, dpn)
        dm = geo.DofManager(xyz.shape[0], dpn)
        idx = np.nonzero(m)[0]
        dm.set_dirichlet(idx, np.repeat(vals, dpn)[idx])
        if dpn == 1:
            K = orc.assemble_thermal_stiffness(xyz, conn, k_e=k_e)
            op = geo.ThermalOperator(mesh, dm, k_e)
        else:
            K = orc.assemble_elasticity_stiffness(xyz, conn, E_e=E_e, nu=0.25)
            op = geo.ElasticityOperator(mesh, dm, geo.IsotropicElasticity(1e11, 0.25), E_e)
        n = dpn * xyz.shape[0]
        f = rng.standard_normal(n)
        Kb, fb = orc.apply_dirichlet_bcs(K, f, m, np.repeat(vals, dpn))
        x = rng.standard_normal(n)
        y = orc.csr_apply(Kb, x)
        # FP64 rounding of the apply; FP32: 2^-24 times the row sums, with room for 30 terms
        for prec, bar in (("fp64", 1e-12), ("mixed", 1e-5)):
            got = op.apply(x, prec)
            assert np.linalg.norm(got - y) <= bar * np.linalg.norm(y), (dpn, prec)
        assert np.linalg.norm(op.lift_rhs(f) - fb) <= 1e-12 * np.linalg.norm(fb), dpn


def test_operators_of_different_sizes(orc, geo):
    """A smaller operator made later leaves the larger one usable, with the same results."""
    box = (1000.0, 1000.0, 600.0)
    ops = []
    for shape in ((12, 11, 10), (2, 1, 1)):
        xyz, conn = orc.generate_cube(*shape, *box)
        # elements in random places: patches with many foreign nodes, so larger tables
        conn = conn[np.random.default_rng(3).permutation(conn.shape[0])]
        xyz = curve(xyz, conn, box, shape)
        mesh = geo.Mesh(xyz, conn)
        for dpn in (1, 3):
            dm = geo.DofManager(xyz.shape[0], dpn)
            op = (geo.ThermalOperator(mesh, dm, 3.0) if dpn == 1 else
                  geo.ElasticityOperator(mesh, dm, geo.IsotropicElasticity(1e11, 0.25)))
            x = np.random.default_rng(5).standard_normal(dpn * xyz.shape[0])
            ops.append((op, x, [op.apply(x, p) for p in ("fp64", "mixed")]))
    for op, x, first in ops:
        for p, y in zip(("fp64", "mixed"), first):
            assert np.array_equal(op.apply(x, p), y)
