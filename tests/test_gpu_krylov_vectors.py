"""The Krylov vector kernels through whole solves at the sizes where they can
go wrong: fewer rows than a warp's tile, remainders of the vector loads, and
more basis vectors than one sweep holds."""

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg

from conftest import has_cuda, rel_err

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]


def _system(n):
    """A nonsymmetric tridiagonal matrix whose unpreconditioned GMRES takes
    most of n steps (eigenvalues spread over [1, 30]), condition below 100."""
    rng = np.random.default_rng(n)
    A = sp.diags([rng.uniform(-0.3, 0.3, n - 1), np.linspace(1.0, 30.0, n), rng.uniform(-0.3, 0.3, n - 1)],
                 [-1, 0, 1], format="csr") if n > 1 else sp.csr_matrix([[3.0]])
    return A, rng.standard_normal(n)


SIZES = [1, 2, 7, 31, 33, 64, 65, 129, 150, 257, 1027]


@pytest.mark.parametrize("n", SIZES)
def test_gmres_sizes(n):
    import torch
    from up3d_b200.solve.linear import solve_gmres
    A, b = _system(n)
    x, n_it, info = solve_gmres(A, torch.from_numpy(b).cuda(), rtol=1e-13, restart=150, maxiter=40, on_fail="return")
    ref = np.linalg.solve(A.toarray(), b)
    # residual 1e-13 |b| times the condition number, and FP64 rounding
    assert info == 0 and rel_err(x.cpu().numpy(), ref) < 1e-10
    if n == 150:
        assert n_it > 64


@pytest.mark.parametrize("n", SIZES)
def test_mixed_gmres_sizes(n):
    import torch
    from up3d_b200.solve.linear import solve_gmres_mixed
    A, b = _system(n)
    x, _, _, info = solve_gmres_mixed(A, torch.from_numpy(b).cuda(), rtol=1e-12, restart=100, maxiter=40,
                                      inner_rtol=1e-5)
    ref = np.linalg.solve(A.toarray(), b)
    assert info == 0 and rel_err(x.cpu().numpy(), ref) < 1e-9


@pytest.mark.parametrize("n", [1, 33, 1023, 1025, 5000])
def test_cg_sizes(n):
    import torch
    from up3d_b200.solve.linear import build_jacobi_preconditioner, solve_cg
    A, b = _system(n)
    A = ((A + A.T) * 0.5).tocsr()
    x, _, info = solve_cg(A, torch.from_numpy(b).cuda(), M=build_jacobi_preconditioner(A), rtol=1e-13, maxiter=500)
    ref = sp.linalg.spsolve(A.tocsc(), b)
    assert info == 0 and rel_err(x.cpu().numpy(), np.atleast_1d(ref)) < 1e-10
