"""The linear algebra at sizes whose kernels the small systems do not reach:
sparse rows in slices and one warp per 32 rows (from 75,776 rows on), and
Krylov vectors of several tiles a block, against scipy."""

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg

from conftest import has_cuda, rel_err
from test_gpu_amg_levels import _hierarchy, _vcycle
from test_gpu_krylov_vectors import _system

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]

SHIFT = 0.05


@pytest.fixture(scope="module", params=["slices", "warp rows"])
def p1(request):
    """A P1 matrix of 81,356 rows (a ragged last slice) with its V-cycle;
    "warp rows": one row of 4,000 more entries, whose padding the slices do
    not take."""
    from up3d_b200.mesh.kuhn import kuhn_box
    nodes, el = kuhn_box(42, 42, 43)
    n, rng = len(nodes), np.random.default_rng(7)
    assert n % 32 and n > 75776
    e = np.vstack([el[:, [i, j]] for i in range(4) for j in range(i)])
    if request.param == "warp rows":
        other = rng.choice(n, size=4000, replace=False)
        e = np.vstack([e, np.column_stack([np.full(4000, n // 2), other])])
    e = np.unique(np.sort(e[e[:, 0] != e[:, 1]], axis=1), axis=0)
    w = rng.uniform(0.5, 2.0, len(e))
    A = sp.coo_matrix((np.r_[-w, -w], (np.r_[e[:, 0], e[:, 1]], np.r_[e[:, 1], e[:, 0]])), shape=(n, n)).tocsr()
    A = (A + sp.diags(SHIFT - np.asarray(A.sum(axis=1)).ravel())).tocsr()
    A.sort_indices()
    length = np.diff(A.indptr)
    padded = 32 * np.maximum.reduceat(length, np.arange(0, n, 32)).sum()
    assert (padded <= A.nnz * 1.125) == (request.param == "slices")
    levels, inv = _hierarchy(A, np.zeros(n, dtype=bool), 500)
    b = rng.standard_normal(n)
    return A, b, levels, inv, _vcycle(levels, inv, b)


def test_products(p1):
    import torch
    from up3d_b200.mesh.device import DeviceCSR
    from up3d_b200.solve.linear import as_device_csr
    A, b, *_ = p1
    Ad = as_device_csr(A)
    scale = abs(A) @ np.abs(b)
    assert (np.abs(Ad.matvec(torch.from_numpy(b).cuda()).cpu().numpy() - A @ b) <= 1e-14 * 4000 * scale).all()
    A32 = DeviceCSR(Ad.indptr, Ad.indices, Ad.data.float(), Ad.shape)
    y = A32.matvec(torch.from_numpy(b).cuda().float()).cpu().numpy()
    assert (np.abs(y - A @ b) <= 6e-8 * 100 * scale).all()      # sums by partial sums of at most 256 entries


@pytest.mark.parametrize("fp32", [False, True])
def test_vcycle(p1, fp32):
    import torch
    from up3d_b200.solve.linear import as_device_csr, build_amg_preconditioner
    A, b, levels, inv, ref = p1
    ml, M = build_amg_preconditioner(as_device_csr(A), fp32=fp32)
    assert ml.n_levels == len(levels) + 1 and ml.n_coarse == len(inv)
    z = M.matvec(torch.from_numpy(b).cuda())
    # rounding amplified by the condition, at most 2 max(diagonal) / SHIFT
    # (about 800, with the long row's 1e4: 2e5)
    cond = 2.0 * A.diagonal().max() / SHIFT
    assert np.abs(z.cpu().numpy() - ref).max() <= (1e-15 * 1e3 if not fp32 else 6e-8) * cond * np.abs(ref).max()
    assert torch.equal(M.matvec(torch.from_numpy(b).cuda()), z)


@pytest.mark.parametrize("fp32", [False, True])
def test_mixed_solve_on_a_cycle_of_either_precision(p1, fp32):
    import torch
    from up3d_b200.solve.linear import as_device_csr, build_amg_preconditioner, solve_gmres_mixed
    A, b, *_ = p1
    Ad = as_device_csr(A)
    M = build_amg_preconditioner(Ad, fp32=fp32)[1]
    x, _, _, info = solve_gmres_mixed(Ad, torch.from_numpy(b).cuda(), M=M, rtol=1e-10, restart=60, maxiter=20)
    r = np.linalg.norm(b - A @ x.cpu().numpy())
    # the test is on the preconditioned residual: its condition (below 100) on top
    assert info == 0 and r <= 1e-8 * np.linalg.norm(b)


N = 130003   # more rows than one tile of every block of a basis sweep, FP64 and FP32


def test_gmres_of_several_tiles():
    import torch
    from up3d_b200.solve.linear import solve_gmres
    A, b = _system(N)
    x, n_it, info = solve_gmres(A, torch.from_numpy(b).cuda(), rtol=1e-13, restart=150, maxiter=40, on_fail="return")
    assert info == 0 and n_it > 64
    # residual 1e-13 |b| times the condition number, and FP64 rounding
    assert rel_err(x.cpu().numpy(), sp.linalg.spsolve(A.tocsc(), b)) < 1e-10


def test_mixed_gmres_of_several_tiles():
    import torch
    from up3d_b200.solve.linear import solve_gmres_mixed
    A, b = _system(N)
    x, n_it, _, info = solve_gmres_mixed(A, torch.from_numpy(b).cuda(), rtol=1e-12, restart=100, maxiter=40,
                                         inner_rtol=1e-6)
    assert info == 0 and n_it > 64
    assert rel_err(x.cpu().numpy(), sp.linalg.spsolve(A.tocsc(), b)) < 1e-9
