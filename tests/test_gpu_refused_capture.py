"""A call that waits for the device is refused inside a stream capture, and
leaves nothing behind: the next call, inside another capture, is taken."""

import numpy as np
import pytest

from conftest import has_cuda

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]


@pytest.mark.parametrize("refused", ["jacobian", "operator", "solve"])
def test_next_call_after_a_refused_one(refused):
    import torch
    from up3d_b200.adjoint import AdjointContext
    from up3d_b200.mesh.kuhn import bump_channel, pocket_state
    from up3d_b200.solve.fused import FlowParams
    from up3d_b200.solve.linear import solve_cg
    from up3d_b200.solve.newton import ChannelWorkspace
    m = bump_channel(8, 4, 5, amplitude=0.08, seed=2)
    ws = ChannelWorkspace(m.nodes, m.elements, m.dirichlet_nodes)
    phi = torch.from_numpy(pocket_state(m, "mixed")).cuda()
    flow = FlowParams(m_inf=0.8)
    actx = AdjointContext(ws, phi, flow)
    lam = torch.from_numpy(np.random.default_rng(0).standard_normal(m.n_nodes)).cuda()
    one = torch.ones(m.n_tets, dtype=torch.float64, device="cuda")
    up = torch.arange(m.n_tets, device="cuda")
    A = ws.picard_matrix()
    call = {"jacobian": lambda: ws.ev.evaluate(phi, flow),
            "operator": lambda: ws.op.assemble_newton_jacobian(phi, one, one, one, up),
            "solve": lambda: solve_cg(A, lam, maxiter=2)}[refused]
    for _ in range(2):
        call()
        dX = actx.vjp(lam=lam)[1]
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError):
        with torch.cuda.graph(torch.cuda.CUDAGraph(), capture_error_mode="thread_local"):
            call()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        out = actx.vjp(lam=lam)[1]
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, dX)
