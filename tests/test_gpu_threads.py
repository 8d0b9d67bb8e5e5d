"""Threads with meshes, hierarchies and streams of their own, side by side:
set-ups, frees, first applications (which capture the cycle) and solves give
the bits that they give alone."""

import threading

import numpy as np
import pytest

from conftest import has_cuda

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]


def _work(k):
    import torch
    from up3d_b200.mesh.device import DeviceMesh
    from up3d_b200.mesh.kuhn import bump_channel, pocket_state
    from up3d_b200.solve.fused import FlowParams, ResidualJacobian
    from up3d_b200.solve.linear import build_amg_preconditioner, solve_cg, solve_gmres_mixed, with_dirichlet
    m = bump_channel(11 + 3 * k, 6, 5, amplitude=0.05, seed=k)
    ev = ResidualJacobian(DeviceMesh(m.nodes, m.elements))
    mask = torch.zeros(m.n_nodes, dtype=torch.uint8, device="cuda")
    mask[torch.from_numpy(m.dirichlet_nodes).cuda()] = 1
    phi = torch.from_numpy(pocket_state(m, "accelerating")).cuda()
    b = torch.sin(torch.arange(m.n_nodes, dtype=torch.float64, device="cuda")).masked_fill(mask.bool(), 0.0)
    out = []
    for _ in range(6):
        ev.evaluate(phi, FlowParams(m_inf=0.5))
        J = with_dirichlet(ev.jacobian(), mask)
        M = build_amg_preconditioner(J, fp32="both", max_coarse=60)[1]
        out += [M.matvec(b), solve_cg(J, b, M=M, rtol=1e-6, maxiter=20)[0],
                solve_gmres_mixed(J, b, M=M, rtol=1e-9, restart=30, maxiter=3)[0]]
        del M
    torch.cuda.current_stream().synchronize()
    return [o.cpu().numpy() for o in out]


def test_threads_side_by_side():
    import torch
    alone = [_work(k) for k in range(4)]
    for _ in range(3):
        got = [None] * 4

        def run(k):
            try:
                with torch.cuda.stream(torch.cuda.Stream()):
                    got[k] = _work(k)
            except Exception as e:   # noqa: BLE001 -- shown by the assertion below
                got[k] = e
        threads = [threading.Thread(target=run, args=(k,)) for k in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for k in range(4):
            assert not isinstance(got[k], Exception), got[k]
            assert all(np.array_equal(a, b) for a, b in zip(got[k], alone[k]))
