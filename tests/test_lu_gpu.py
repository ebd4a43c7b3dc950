"""The FP64 LU with partial pivoting at the sizes where its kernels change
shape: one step and several (64 columns each), sub-panels of 16 and 8 columns,
one to eight rows per thread (512, 1024, 1536, 2048 rows), ragged last steps."""
import numpy as np
import pytest

from adga_b200 import inverse_matrix

SIZES = [1, 2, 7, 8, 15, 16, 17, 31, 33, 40, 63, 64, 65, 79, 80, 128, 129, 357, 511, 512, 513, 577, 1024, 1025, 1089,
         1537, 2049]


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
def test_inverse_residual(n):
    """Backward-stable elimination: |X A - 1|_2 <= c n eps cond(A) with a
    modest growth factor in c (32)."""
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(2 * n)
    X, ierr, _ = inverse_matrix(A)
    assert ierr == 0
    s = np.linalg.svd(A, compute_uv=False)
    tol = 32 * n * np.finfo(float).eps * s[0] / s[-1]
    assert np.linalg.norm(X @ A - np.eye(n), 2) <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
def test_inverse_of_signed_permutation_is_exact(n):
    """Every pivot is far from the diagonal and every operation is exact."""
    rng = np.random.default_rng(1000 + n)
    A = np.zeros((n, n), dtype=complex)
    A[np.arange(n), rng.permutation(n)] = rng.choice([1, -1, 1j, -1j], n) * 2.0 ** rng.integers(-40, 40, n)
    X, ierr, _ = inverse_matrix(A)
    assert ierr == 0
    want = np.zeros_like(A)
    r, c = np.nonzero(A)
    want[c, r] = A[r, c].conj() / np.abs(A[r, c]) ** 2
    assert np.array_equal(X, want)


@pytest.mark.gpu
@pytest.mark.parametrize("n,col", [(1, 0), (40, 17), (64, 63), (65, 64), (200, 130), (600, 5), (1030, 1029)])
def test_zero_column_is_reported(n, col):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A[:, col] = 0.0
    assert inverse_matrix(A)[1] == col + 1


@pytest.mark.gpu
@pytest.mark.parametrize("n,at", [(1, 0), (5, 2), (40, 0), (64, 63), (80, 41), (81, 7), (130, 129), (357, 64), (600, 300),
                                  (1030, 1029)])
def test_infinite_pivot_drops_its_row_and_column(n, at):
    """The reciprocal of an infinite pivot is zero (Smith's division): the
    inverse is that of the matrix without the row and the column, zeros in their
    place.  Diagonally dominant, so that the row is no earlier column's pivot;
    error bound as above, with growth 1 and condition 2."""
    rng = np.random.default_rng(n)
    A = (rng.uniform(-1, 1, (n, n)) + 1j * rng.uniform(-1, 1, (n, n))) / (6 * n) + np.eye(n)
    keep = np.arange(n) != at
    want = np.zeros_like(A)
    want[np.ix_(keep, keep)] = np.linalg.inv(A[np.ix_(keep, keep)])
    A[at, at] = complex(np.inf, 0.5)
    X, ierr, _ = inverse_matrix(A)
    assert ierr == 0
    assert np.max(np.abs(X - want)) <= 32 * n * np.finfo(float).eps * 2


@pytest.mark.gpu
@pytest.mark.parametrize("n", [40, 100, 520, 1030])
def test_column_of_nan_reaches_the_columns_after_it(n):
    """No row of the column can be a pivot; its multipliers make the columns
    after it NaN too, the zero one among them, which then is no zero pivot."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    assert inverse_matrix(A)[1] == 0         # leaves finite values where the kernel keeps its rows
    A[:, 1] = np.nan
    A[:, 2] = 0.0
    X, ierr, _ = inverse_matrix(A)
    assert ierr == 0
    assert np.isnan(X.real).all()
