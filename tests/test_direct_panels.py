"""The blocked LU at the edges of its panels, tiles and look-ahead: sizes around the panel
width (32; 16 above 4096 rows, 8 above 8192), the 64-column tiles, one to eight blocks per
cluster and the first size with look-ahead. Rows rolled so that nearly every column pivots
far from the diagonal. Against scipy's sparse LU."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 96, 127, 129, 513, 640, 641, 705, 1025, 2049, 4097, 8225])
def test_panel_edges(geo, n):
    import scipy.sparse as sp
    import scipy.sparse.linalg as spl
    rng = np.random.default_rng(n)
    M = sp.diags([4.0 + rng.random(n)], [0]).tocsr()
    if n > 1:
        M = M + sp.diags([-1.3 * np.ones(n - 1), -0.7 * np.ones(n - 1)], [-1, 1])
        M = M + 0.1 * sp.random(n, n, density=min(0.2, 4.0 / n), random_state=n)
    M = M.tocsr()[np.roll(np.arange(n), n // 3)].tocsr()
    M.sort_indices()
    b = rng.standard_normal(n)
    x, st = geo.DirectSolver().solve(geo.CsrMatrix.from_arrays(n, n, M.indptr, M.indices, M.data), b)
    xs = np.atleast_1d(spl.spsolve(M.tocsc(), b))
    # condition number below 10: the LU's backward error times it, with a wide margin
    assert np.linalg.norm(x - xs) <= 1e-12 * np.linalg.norm(xs)
    assert st.converged and st.relative_residual <= 1e-13
