"""The AMG's dense coarsest inverse where the pivots decide: rows that have to
change places, one size beside each panel and cluster form, a singular matrix
(regularised), an infinity and NaN (in the result, not in the way)."""

import numpy as np
import pytest
import scipy.sparse as sp

from conftest import has_cuda

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]

SIZES = [1, 2, 7, 8, 9, 16, 17, 129, 500, 512, 513]


def _apply(A, b):
    import torch
    from up3d_b200.solve.linear import build_amg_preconditioner
    ml, M = build_amg_preconditioner(A, max_coarse=600)
    assert ml.n_coarse == A.shape[0]
    return M.matvec(torch.from_numpy(b).cuda()).cpu().numpy()


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", ["reversed", "shuffled", "graded"])
def test_rows_change_places(n, kind):
    rng = np.random.default_rng(n)
    A = np.diag(rng.uniform(1.0, 2.0, n)) + rng.uniform(-0.2, 0.2, (n, n)) / n
    if kind == "graded":
        A *= 10.0 ** rng.integers(-3, 4, n)[:, None]
    A = A[::-1] if kind == "reversed" else A[rng.permutation(n)]
    b = rng.standard_normal(n)
    z, ref = _apply(sp.csr_matrix(A), b), np.linalg.solve(A, b)
    # condition below 1e7 (graded), n rounding errors per entry
    assert np.abs(z - ref).max() <= 1e-16 * n * (1e7 if kind == "graded" else 10.0) * np.abs(ref).max() + 1e-15


@pytest.mark.parametrize("n", [2, 9, 129, 512, 513])
def test_singular_matrix_is_regularised(n):
    A = sp.diags([-np.ones(n - 1), np.r_[1.0, np.full(n - 2, 2.0), 1.0], -np.ones(n - 1)], [-1, 0, 1]).tocsr()
    b = np.random.default_rng(n).standard_normal(n)
    b -= b.mean()
    z = _apply(A, b)
    assert np.isfinite(z).all()
    # n^2 / 10 bounds the inverse off the null space; the shift adds its share of it
    assert np.abs(A @ z - b).max() < 1e-3 * np.abs(b).max()


@pytest.mark.parametrize("n", [2, 9, 129, 512, 513])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_not_finite_entries_end_in_the_result(n, value):
    A = np.diag(np.full(n, 2.0)) + np.diag(np.full(n - 1, -0.5), 1) + np.diag(np.full(n - 1, -0.5), -1)
    A[n // 2, n // 2] = value
    z = _apply(sp.csr_matrix(A), np.ones(n))
    if np.isnan(value):
        assert np.isnan(z).any()
    else:                                   # the row's reciprocal is 0: inf * 0
        assert not np.isfinite(z).all() or np.abs(z[n // 2]) < 1e-300
