"""The finest operator of an AMG hierarchy (identity rows and no columns at
constrained DOFs), through a hierarchy of one level, whose V-cycle is the
dense solve with it: row lengths around the lanes that copy a row, rows of
the diagonal only, no, some and all DOFs constrained."""

import numpy as np
import pytest
import scipy.sparse as sp

from conftest import has_cuda

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]


@pytest.mark.parametrize("n", [1, 7, 33, 300])
@pytest.mark.parametrize("constrained", [None, "none", "some", "all"])
def test_one_level_hierarchy_solves_the_embedded_system(n, constrained):
    import torch
    from up3d_b200.kernels.jacobian import DeviceCSR
    from up3d_b200.solve.linear import build_amg_preconditioner
    rng = np.random.default_rng(n)
    A = sp.lil_matrix((n, n))
    for r in range(n):
        k = min(n, int(rng.choice([1, 7, 8, 9, 17, 60])))
        cols = np.unique(np.append(rng.choice(n, size=k, replace=False), r))
        A[r, cols] = rng.uniform(-1.0, 1.0, len(cols))
        A[r, r] = len(cols) + 1.0           # diagonally dominant: well conditioned
    A = sp.csr_matrix(A)
    A.sort_indices()
    skip = {None: np.zeros(n, bool), "none": np.zeros(n, bool), "some": rng.random(n) < 0.3,
            "all": np.ones(n, bool)}[constrained]
    E = A.toarray()
    E[skip, :] = 0.0
    E[:, skip] = 0.0
    E[skip, skip] = 1.0
    b = rng.standard_normal(n)
    want = np.linalg.solve(E, b)
    cuda = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in
            (A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data)]
    mask = None if constrained is None else torch.from_numpy(skip.astype(np.uint8)).cuda()
    M = build_amg_preconditioner(DeviceCSR(*cuda, (n, n)), dirichlet=mask, max_coarse=500)[1]
    got = M.matvec(torch.from_numpy(b).cuda()).cpu().numpy()
    # condition below 100 and growth of the explicit inverse: 300 eps each
    assert np.abs(got - want).max() <= 1e-11 * np.abs(want).max()
