"""The dense LU on matrices with infinities and NaN: a NaN is never a pivot (a column with
nothing else left is singular), and a zero multiplier takes no part in a product with an
infinity or a NaN. Against the elimination written out in numpy, at sizes with one and with
several panels, tiles and look-ahead."""
import numpy as np
import pytest


def eliminate(M, b):
    """Partial pivoting, first largest |a_ik|, rows with a zero multiplier left alone; None
    when it meets a column without a pivot."""
    with np.errstate(all="ignore"):
        A = np.column_stack([M, b]).astype(float)
        n = M.shape[0]
        for k in range(n):
            key = np.where(np.isnan(A[k:, k]), 0.0, np.abs(A[k:, k]))
            p = k + int(np.argmax(key))
            if key[p - k] == 0.0:
                return None
            A[[k, p]] = A[[p, k]]
            l = A[k + 1:, k] / A[k, k]
            rows = k + 1 + np.nonzero(l != 0.0)[0]  # NaN != 0
            A[rows, k + 1:] -= l[rows - k - 1, None] * A[k, None, k + 1:]
        x = np.zeros(n)
        for r in range(n - 1, -1, -1):
            x[r] = (A[r, n] - A[r, r + 1:n] @ x[r + 1:]) / A[r, r]
        return x


def matrix(kind, n):
    rng = np.random.default_rng(n)
    M = rng.standard_normal((n, n)) + n * np.eye(n)
    if kind == "band":
        M[np.abs(np.subtract.outer(np.arange(n), np.arange(n))) > 3] = 0.0
    if kind == "triangle":
        M = np.triu(M)
    return M, rng.standard_normal(n)


def places(n):
    if n > 200:
        return [(0, n - 1), (n // 2, n // 3)]
    return sorted({(0, 0), (0, n - 1), (n - 1, 0), (n - 1, n - 1), (n // 2, n // 3), (n // 3, n // 2)})


def test_elimination_written_out():
    for kind in ("dense", "band", "triangle"):
        M, b = matrix(kind, 40)
        assert np.allclose(eliminate(M, b), np.linalg.solve(M, b), rtol=1e-12, atol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("kind", ["dense", "band", "triangle"])
@pytest.mark.parametrize("n", [1, 2, 3, 20, 33, 70, 150, 705])
def test_nonfinite_entry(geo, n, kind, value):
    for i, j in places(n):
        M, b = matrix(kind, n)
        M[i, j] = value
        ref = eliminate(M, b)
        A = geo.CsrMatrix.from_arrays(n, n, np.arange(n + 1) * n, np.tile(np.arange(n), n), M.ravel())
        if ref is None:
            with pytest.raises(geo.GeoError, match="singular"):
                geo.DirectSolver().solve(A, b)
            continue
        x, st = geo.DirectSolver().solve(A, b)
        with np.errstate(all="ignore"):
            assert np.array_equal(np.isfinite(x), np.isfinite(ref)), (i, j)
            ok = np.isfinite(ref)
            # condition number below 10 where the entry is not part of it
            assert np.abs(x - ref)[ok].max(initial=0.0) <= 1e-11 * np.abs(ref[ok]).max(initial=0.0), (i, j)
        if not ok.all():
            assert not st.converged
