"""The CSR PCG's two forms at their edges: matrices that fill a few warps, blocks of 256, 512
and 1024 threads, one pass of the grid less or more than one row, rows longer than a step,
empty blocks. Against the oracle's restated loop (equal iteration counts within the
rounding of the sums, solutions to the tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def spd(n, seed, dense_row):
    import scipy.sparse as sp
    rng = np.random.default_rng(seed)
    A = sp.diags([4.0 + rng.random(n)], [0]).tolil()
    if n > 1:
        A.setdiag(-1.0, 1)
        A.setdiag(-1.0, -1)
    if dense_row and n > 40:
        c = rng.choice(np.arange(2, n), size=min(n - 2, 600), replace=False)
        A[0, c] = -1e-3
        A[c, 0] = -1e-3
    A = A.tocsr()
    A.sort_indices()
    return A, rng.standard_normal(n)


@pytest.mark.parametrize("n", [1, 2, 7, 63, 64, 65, 257, 9471, 9473, 18945, 37887, 37888, 37889, 40001])
def test_sizes_against_oracle(orc, geo, n):
    A, b = spd(n, n, n % 2 == 1)
    Ao = orc.Csr(n, n, A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data.astype(np.float64))
    xo, so = orc.cg_solve(Ao, b, 1000, 1e-10)
    x, st = geo.ConjugateGradient().with_tolerance(1e-10).solve(
        geo.CsrMatrix.from_arrays(n, n, A.indptr, A.indices, A.data), b)
    assert st.converged and abs(st.iterations - so.iterations) <= 1
    assert np.linalg.norm(x - xo) <= 1e-9 * np.linalg.norm(xo)
    assert np.linalg.norm(A @ x - b) <= 2e-10 * np.linalg.norm(b)
