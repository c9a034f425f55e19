"""Linear solves whose matrices the natural order solves without pivoting but another
order may not: rows with a zero or tiny diagonal entry, which the natural order meets
after their neighbours have filled it in.  gf_band_solve and gf_sparse_solve accept the
multifrontal LU's solution where every row's residual is within 2^-49 (sum_j |a_ij| max_j
|x_j| + |b_i|), else the natural order's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def row_error(A, x, b):
    """Largest residual of a row over its denominator, the sums in long double."""
    A = A.astype(np.longdouble)
    r = np.abs(b - A @ x)
    d = np.abs(A).sum(1) * np.where(A != 0, np.abs(x), 0).max(1) + np.abs(b)
    return float((r / d).max())


def gb(A, kl, ku):
    n = len(A)
    ab = np.full((n, 2 * kl + ku + 1), np.nan)
    for j in range(n):
        i = np.arange(max(0, j - ku), min(n, j + kl + 1))
        ab[j, kl + ku + i - j] = A[i, j]
    return ab


@pytest.mark.parametrize("weak", [0.0, 1e-14, 1e-9, 1e-6, 1e-3])
@pytest.mark.parametrize("row", [12, 24, 36, 37, 48])
def test_tridiagonal_with_a_weak_row(gpu_ctx, row, weak):
    # blocks of 12: every block that a separator precedes starts with this row
    n = 60
    A = 2.0 * np.eye(n) + np.eye(n, k=1) * 0.9 + np.eye(n, k=-1) * 0.9
    A[row, row] = weak
    b = np.random.default_rng(7).normal(size=n)
    ab = gb(A, 1, 1)
    x, info = gpu_ctx.band_solve(ab, 1, 1, b)
    # both ways: the accepted solution by the limit, the natural order's pivots grow by
    # at most 1 + |a|^2 / |pivot| < 16
    assert info == 0 and row_error(A, x, b) <= 2.0 ** -49
    y, info = gpu_ctx.band_solve_noalloc(np.nan_to_num(ab), 1, 1, b)
    # each within the limit: the forward error is the inverse's rows times it
    d = np.abs(A).sum(1) * np.abs(x).max() + np.abs(b)
    assert info == 0 and np.abs(x - y).max() <= 2 * 2.0 ** -49 * (np.abs(np.linalg.inv(A)) @ d).max()


@pytest.mark.parametrize("row", list(range(12, 240, 12)))
def test_band_with_a_weak_row(gpu_ctx, row):
    # the natural order's pivot of the row is about 1 / 16 of its couplings: 16 x 16
    # roundings where its solution is the one returned
    n, w = 240, 5
    i = np.arange(n)
    A = np.where(np.abs(i[:, None] - i[None, :]) <= w, np.random.default_rng(row).uniform(-1.0, 1.0, (n, n)), 0.0)
    A[i, i] = 1.5 * (2 * w + 1)
    A[row, row] = 1e-12
    A[row, row - 1] = A[row - 1, row] = 1.0
    b = np.random.default_rng(7).normal(size=n)
    x, info = gpu_ctx.band_solve(gb(A, w, w), w, w, b)
    assert info == 0 and row_error(A, x, b) <= 2.0 ** -45


@pytest.mark.parametrize("weak", [0.0, 1e-13])
def test_grid_with_a_weak_row(gpu_ctx, weak):
    g = 30
    n = g * g
    T = np.eye(g) + np.eye(g, k=1) + np.eye(g, k=-1)
    M = np.kron(T, T) != 0
    A = np.where(M, np.random.default_rng(0).uniform(-1.0, 1.0, (n, n)), 0.0)
    np.fill_diagonal(A, 0.0)
    np.fill_diagonal(A, 1.5 * np.abs(A).sum(1) + 0.1)
    b = np.random.default_rng(1).normal(size=n)
    rows, cols = np.nonzero(M)
    rp = np.concatenate([[0], np.cumsum(M.sum(1))]).astype(np.int32)
    for r in range(g + 1, n, 5):
        B = A.copy()
        B[r, r] = weak
        x, info = gpu_ctx.sparse_solve(rp, cols.astype(np.int32), B[rows, cols], b)
        # the band's order fills the row in from the row of the grid before it (couplings
        # of up to 1 on diagonals of 3 to 8: a pivot of 1 / 16 or so)
        assert info == 0, r
        res, d = np.abs(b - B @ x), np.abs(B).sum(1) * np.abs(x).max() + np.abs(b)
        assert (res / d).max() <= 2.0 ** -44, r


@pytest.mark.parametrize("g,shift", [(100, 0.0), (60, 0.37)])
def test_refinement_on_the_fronts(gpu_ctx, g, shift):
    # five-point Laplacians, one of them indefinite: the tensor-core products leave rows of 36
    # and 6,000 roundings, refined with the factor to within the limit
    n = g * g
    at = np.arange(n)
    cols = np.stack([at - g, at - 1, at, at + 1, at + g], axis=1)
    live = np.stack([at >= g, at % g > 0, at >= 0, at % g < g - 1, at < n - g], axis=1)
    vals = np.where(np.arange(5) == 2, 4.0 - shift, -1.0) * live
    b = np.random.default_rng(5).normal(size=n)
    rp = np.concatenate([[0], np.cumsum(live.sum(1))]).astype(np.int32)
    x, info = gpu_ctx.sparse_solve(rp, cols[live].astype(np.int32), vals[live], b)
    xc = np.where(live, x[np.clip(cols, 0, n - 1)], 0.0).astype(np.longdouble)
    r = np.abs(b - (vals * xc).sum(1))
    d = np.abs(vals).sum(1) * np.abs(xc).max(1) + np.abs(b)
    # the limit, and the residual's own five roundings
    assert info == 0 and float((r / d).max()) <= 2.0 ** -49 + 5 * 2.0 ** -53
