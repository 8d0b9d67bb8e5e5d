"""The adjoint's upstream sums for weights of either sign: the residual's
vector-Jacobian product is linear and odd in lambda, so -lambda gives the
negated gradients bit for bit, also where a chain of elements upstream sums
to a negative weight."""

import numpy as np
import pytest

from conftest import has_cuda

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]


@pytest.mark.parametrize("shared", [1, 40, 400])   # chains of 840, 21 and 2 or 3 elements
@pytest.mark.parametrize("gamma", [1.4, 1.3])
def test_negated_lambda_negates_the_gradients(shared, gamma):
    import torch
    from up3d_b200.adjoint import AdjointContext
    from up3d_b200.mesh.kuhn import bump_channel, pocket_state
    from up3d_b200.solve.fused import FlowParams
    from up3d_b200.solve.newton import ChannelWorkspace
    mesh = bump_channel(7, 4, 5, amplitude=0.05, seed=3)
    E = mesh.n_tets
    rng = np.random.default_rng(shared)
    up = rng.choice(E, size=shared, replace=False)[np.arange(E) % shared]
    branch = np.where(up == np.arange(E), 0, 1 + np.arange(E) % 2).astype(np.int8)
    phi = torch.from_numpy(pocket_state(mesh, "accelerating")).cuda()
    lam = torch.from_numpy(rng.standard_normal(mesh.n_nodes)).cuda()
    actx = AdjointContext(ChannelWorkspace(mesh.nodes, mesh.elements, mesh.dirichlet_nodes), phi,
                          FlowParams(m_inf=0.8, gamma=gamma),
                          frozen=(torch.from_numpy(up).cuda(), torch.from_numpy(branch).cuda()))
    plus, minus = actx.vjp(lam=lam)[1:], actx.vjp(lam=-lam)[1:]
    for p, m in zip(plus, minus):
        assert torch.equal(p, -m) and bool(torch.isfinite(p).all())
