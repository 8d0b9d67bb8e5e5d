"""The FP32 cycle on the caller's FP64 vectors converts in the sweeps that
read and write them: no launch more than the FP64 cycle makes."""

import numpy as np
import pytest

from conftest import has_cuda

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]


def _launches(M, x):
    import ctypes
    from up3d_b200 import _lib as L
    n = [ctypes.c_int64(), ctypes.c_int64()]
    M.matvec(x)                              # the captured body
    L.call("up3d_launch_count", ctypes.byref(n[0]))
    z = M.matvec(x)
    L.call("up3d_launch_count", ctypes.byref(n[1]))
    return n[1].value - n[0].value, z


@pytest.mark.parametrize("post", [0, 1, 2])
def test_fp32_cycle_takes_no_more_launches(post):
    import scipy.sparse as sp
    import torch
    from up3d_b200.solve.linear import build_amg_preconditioner
    n = 3001
    A = (sp.diags([-1.0, 2.05, -1.0], [-1, 0, 1], shape=(n, n))).tocsr()
    x = torch.from_numpy(np.random.default_rng(0).standard_normal(n)).cuda()
    l64, z64 = _launches(build_amg_preconditioner(A, postsmooth=post)[1], x)
    l32, z32 = _launches(build_amg_preconditioner(A, fp32=True, postsmooth=post)[1], x)
    assert l32 == l64 if post else l32 <= l64 + 1     # without a last sweep: a conversion in place of a copy
    # FP32 rounding times the condition (4.05 / 0.05)
    assert float((z32 - z64).abs().max()) < 1e-4 * float(z64.abs().max())
