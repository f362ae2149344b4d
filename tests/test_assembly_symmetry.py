"""The assembled matrices are symmetric to rounding, and the sums of the element matrices
that the element routines return. K_ij and K_ji, and the element routines, form the same
terms by different expressions; a term takes some 60 operations and an entry sums at most
4 points of some 24 elements, all bounded by the row's scale: 64 units in the last place."""
import numpy as np
import pytest

from test_golden import row_err

pytestmark = pytest.mark.gpu

BAR = 64 * 2.0 ** -53


@pytest.mark.parametrize("curved", [False, True])
@pytest.mark.parametrize("dpn", [1, 3])
def test_symmetric_sums_of_element_matrices(orc, geo, dpn, curved):
    xyz, conn = orc.generate_cube(9, 8, 7, 1.0, 1.2, 0.8)
    rng = np.random.default_rng(1)
    if curved:
        nv = np.unique(conn[:, :4]).size
        xyz = xyz.copy()
        xyz[nv:] += rng.uniform(-0.01, 0.01, (xyz.shape[0] - nv, 3))
    coef = rng.uniform(0.5, 4.0, conn.shape[0])
    mesh, dm = geo.Mesh(xyz, conn), geo.DofManager(xyz.shape[0], dpn)
    mat = geo.IsotropicElasticity(1.0, 0.25)
    if dpn == 1:
        K = geo.Assembler.assemble_thermal_stiffness_parallel(mesh, dm, coef)
        Ke = geo.ElementMatrix.thermal_stiffness(mesh, coef)
    else:
        K = geo.Assembler.assemble_elasticity_stiffness_parallel(mesh, dm, mat, coef)
        Ke = geo.ElasticityElement.stiffness_matrix(mesh, mat, coef)
    ip, ix, data = K.to_host()
    import scipy.sparse as sp
    A = sp.csr_matrix((data, ix, ip))
    T = A.T.tocsr()
    T.sort_indices()
    assert row_err(T.data, data, ip) <= BAR
    dofs = (dpn * conn[:, :, None] + np.arange(dpn)).reshape(conn.shape[0], -1)
    S = sp.coo_matrix((np.asarray(Ke).reshape(-1), (np.repeat(dofs, dofs.shape[1], axis=1).reshape(-1),
                                                    np.tile(dofs, (1, dofs.shape[1])).reshape(-1))), A.shape).tocsr()
    S.sort_indices()
    assert np.array_equal(S.indptr, ip) and np.array_equal(S.indices, ix)
    assert row_err(S.data, data, ip) <= BAR
