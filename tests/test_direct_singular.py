"""Singular matrices with the zero pivot in the first, a middle and the last panel, with and
without look-ahead (panels, pivot rows and trailing tiles of two panels in flight): refused,
and the next solve of a regular matrix is as if nothing had happened."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dense(geo, M):
    n = M.shape[0]
    return geo.CsrMatrix.from_arrays(n, n, np.arange(n + 1) * n, np.tile(np.arange(n), n), M.ravel())


@pytest.mark.parametrize("n", [150, 705, 2049])
def test_zero_column(geo, n):
    rng = np.random.default_rng(n)
    M = rng.standard_normal((n, n))
    b = rng.standard_normal(n)
    regular = dense(geo, M)
    first, _ = geo.DirectSolver().solve(regular, b)
    for c in sorted({0, 31, 32, 95, n // 2, n - 33, n - 2, n - 1}):
        S = M.copy()
        S[:, c] = 0.0  # stays zero under elimination
        with pytest.raises(geo.GeoError, match="singular"):
            geo.DirectSolver().solve(dense(geo, S), b)
    again, _ = geo.DirectSolver().solve(regular, b)
    assert np.array_equal(first, again)
