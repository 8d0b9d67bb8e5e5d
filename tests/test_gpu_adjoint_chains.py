"""The adjoint's per-upstream sums on chains of every length: one element
upstream of all the others, a few shared ones, and none, against central
finite differences of the residual at that (frozen) selection; and the same
bits on every call, whatever order the chains were built in."""

import numpy as np
import pytest

from conftest import has_cuda

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]


@pytest.mark.parametrize("shared", [1, 5, 0])
@pytest.mark.parametrize("gamma", [1.4, 1.3])
def test_chains_match_finite_differences(shared, gamma):
    import torch
    from up3d_b200.adjoint import AdjointContext
    from up3d_b200.mesh.kuhn import bump_channel, pocket_state
    from up3d_b200.solve.fused import FlowParams
    from up3d_b200.solve.newton import ChannelWorkspace
    mesh = bump_channel(7, 4, 5, amplitude=0.05, seed=3)
    E = mesh.n_tets
    rng = np.random.default_rng(shared)
    up = np.arange(E)
    if shared:
        up = rng.choice(E, size=shared, replace=False)[np.arange(E) % shared]
    own = up == np.arange(E)
    branch = np.where(own, 0, 1 + np.arange(E) % 2).astype(np.int8)
    flow = FlowParams(m_inf=0.8, gamma=gamma)
    phi = torch.from_numpy(pocket_state(mesh, "accelerating")).cuda()
    lam = torch.from_numpy(rng.standard_normal(mesh.n_nodes)).cuda()
    frozen = (torch.from_numpy(up).cuda(), torch.from_numpy(branch).cuda())

    def value(nodes, flow=flow):
        ws = ChannelWorkspace(nodes, mesh.elements, mesh.dirichlet_nodes)
        return float(lam @ ws.ev.evaluate(phi, flow, jacobian=False, frozen=frozen, keep_state=False))

    actx = AdjointContext(ChannelWorkspace(mesh.nodes, mesh.elements, mesh.dirichlet_nodes), phi, flow, frozen=frozen)
    _, dX, dM = actx.vjp(lam=lam)
    _, dX2, dM2 = actx.vjp(lam=lam)
    assert torch.equal(dX, dX2) and torch.equal(dM, dM2)
    # central differences: h^2 truncation and rounding / h, both far below 1e-6
    h = 1e-6
    d = rng.standard_normal(mesh.nodes.shape)
    fd = (value(mesh.nodes + h * d) - value(mesh.nodes - h * d)) / (2 * h)
    ad = float((dX.cpu().numpy() * d).sum())
    assert abs(fd - ad) <= 1e-6 * abs(ad)
    fd = (value(mesh.nodes, FlowParams(m_inf=0.8 + h, gamma=gamma))
          - value(mesh.nodes, FlowParams(m_inf=0.8 - h, gamma=gamma))) / (2 * h)
    assert abs(fd - float(dM)) <= 1e-6 * abs(float(dM))
