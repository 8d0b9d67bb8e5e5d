"""The fused element sweep where an element and its upstream one are surely
below the critical speed (their switch is 0 and is not formed), against the
per-element kernels that form it everywhere: speeds below, across and at the
critical one, floored densities, no critical speed (M_inf or M_crit 0), air
and another gas, element counts that end inside a warp, every launch shape."""

import numpy as np
import pytest

from conftest import REL_TOL, has_cuda, rel_err, sparse_rel_err

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]

SHAPES = [(0, 512), (1, 512), (1, 640), (0, 768), (1, 768)]


def _critical_q2(m_inf, m_crit, gamma):
    h = 0.5 * (gamma - 1.0)
    return m_crit ** 2 * (1.0 + h * m_inf ** 2) / (m_inf ** 2 * (1.0 + h * m_crit ** 2))


@pytest.mark.parametrize("cells", [(1, 1, 1), (3, 3, 3), (15, 5, 7)])
@pytest.mark.parametrize("gamma", [1.4, 1.3])
@pytest.mark.parametrize("m_inf,m_crit,floor,speed", [
    (0.8, 0.95, 0.05, "below"), (0.8, 0.95, 0.05, "across"), (0.8, 0.95, 0.05, "at"), (0.8, 0.95, 0.99, "across"),
    (0.8, 0.95, 0.99, "below"), (0.0, 0.95, 0.05, "below"), (0.8, 0.0, 0.05, "below")])
def test_against_the_kernels_that_form_every_switch(cells, gamma, m_inf, m_crit, floor, speed):
    import torch
    from up3d_b200.kernels.jacobian import PicardOperator
    from up3d_b200.kernels.upwind import UpwindOperator
    from up3d_b200.mesh.device import DeviceMesh
    from up3d_b200.mesh.kuhn import bump_channel
    from up3d_b200.physics.isentropic import density_field, limit_q2_field
    from up3d_b200.solve.fused import FlowParams, ResidualJacobian
    mesh = bump_channel(*cells, amplitude=0.05, seed=1)
    assert mesh.n_tets % 32 != 0
    rng = np.random.default_rng(cells[0])
    crit = _critical_q2(0.8, 0.95, gamma)
    noise = {"below": 0.004, "across": 0.02, "at": 1e-15}[speed]
    u = np.sqrt(crit) * {"below": 0.8, "across": 0.99, "at": 1.0}[speed]
    phi_h = u * mesh.nodes[:, 0] + noise * rng.standard_normal(len(mesh.nodes))
    phi = torch.from_numpy(phi_h).cuda()
    flow = FlowParams(m_inf=m_inf, gamma=gamma, m_crit=m_crit, rho_floor=floor)

    nodes, elements = torch.from_numpy(mesh.nodes), torch.from_numpy(mesh.elements)
    op, upw = PicardOperator(nodes, elements), UpwindOperator(nodes, elements)
    grad, q2 = op.velocities(phi)
    q2l = limit_q2_field(q2, m_inf, flow.m_cap, gamma)
    rho = density_field(q2l, m_inf, gamma)
    args = (grad, q2l, rho, m_inf, flow.upwind_c, m_crit, gamma, floor)
    rt = upw.rho_tilde(*args).clone()
    sup, flo = upw.n_supersonic, upw.n_floored
    se, su, up = upw.rho_tilde_sensitivities(*args)
    R = op.assemble_residual(phi, rt).cpu().numpy()
    J = op.assemble_newton_jacobian(phi, rt, se, su, up, lim_mask=q2l == q2)

    dm = DeviceMesh(mesh.nodes, mesh.elements)
    ev = ResidualJacobian(dm)
    for shape in SHAPES:
        dm.set_tuning(*shape)
        got = ev.evaluate(phi, flow).cpu().numpy()
        mon = ev.read_monitors()
        assert torch.equal(ev.upstream.to(torch.int64), up.to(torch.int64))
        assert rel_err(ev.rho_tilde.cpu().numpy(), rt.cpu().numpy()) < 1e-14
        assert rel_err(got, R) < REL_TOL
        assert sparse_rel_err(ev.jacobian().to_scipy(), J.to_scipy()) < REL_TOL
        assert (mon["n_supersonic"], mon["n_floored"]) == (sup, flo)
        only = ev.evaluate(phi, flow, jacobian=False).cpu().numpy()
        assert np.array_equal(only, got)


@pytest.mark.parametrize("gammas", [(1.4, 1.4), (1.4, 1.3), (1.3, 1.3)])
def test_captured_batch_follows_a_new_flow_table(gammas):
    """A captured evaluation reads the flow table of its replay, also when
    the gas is another than the one it was captured with."""
    import torch
    from up3d_b200 import _lib as L
    from up3d_b200.mesh.kuhn import bump_channel
    from up3d_b200.solve.batched import BatchedChannels
    from up3d_b200.solve.fused import FlowParams
    meshes = [bump_channel(6, 3, 3, amplitude=0.05, seed=k) for k in range(2)]
    batch = BatchedChannels(meshes)
    rng = np.random.default_rng(3)
    x = np.concatenate([m.nodes[:, 0] for m in meshes])
    phi = torch.from_numpy(1.1 * x + 0.02 * rng.standard_normal(len(x))).cuda()
    batch.evaluate(phi, [0.8, 0.7], jacobian=False)          # air
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        batch.evaluate(phi, None, jacobian=False)
        graph.capture_begin()
        try:
            batch.evaluate(phi, None, jacobian=False)
        finally:
            graph.capture_end()
    torch.cuda.current_stream().wait_stream(side)
    flows = (L.Flow * 2)(*[FlowParams(m_inf=m, gamma=g).c() for m, g in zip((0.8, 0.7), gammas)])
    batch._flows = lambda machs: flows
    direct = batch.evaluate(phi, [0.8, 0.7], jacobian=False).clone()
    batch.ws.ev.R.zero_()
    graph.replay()
    torch.cuda.synchronize()
    scale = direct.abs().max()
    assert float((batch.ws.ev.R - direct).abs().max()) <= 1e-14 * float(scale)
