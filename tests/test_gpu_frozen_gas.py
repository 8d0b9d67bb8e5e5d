"""The frozen sweep of air and of another gas, which forms every pair's switch:
elements left live (branch -1) keep the bits of the live sweep, whole and in
part, and the selection frozen at a state gives that state's evaluation."""

import numpy as np
import pytest

from conftest import REL_TOL, has_cuda, rel_err, sparse_rel_err

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]


@pytest.mark.parametrize("gamma", [1.4, 1.3])
@pytest.mark.parametrize("threads,persistent", [(512, 0), (640, 1), (768, 0), (768, 1)])
def test_frozen_sweep_keeps_live_bits(gamma, threads, persistent):
    import torch
    from up3d_b200.mesh.kuhn import bump_channel, pocket_state
    from up3d_b200.solve.fused import FlowParams
    from up3d_b200.solve.newton import ChannelWorkspace
    m = bump_channel(13, 5, 7, amplitude=0.08, seed=2)
    ws = ChannelWorkspace(m.nodes, m.elements, m.dirichlet_nodes)
    phi = torch.from_numpy(pocket_state(m, "mixed")).cuda()
    flow = FlowParams(m_inf=0.8, gamma=gamma)
    ws.ev.mesh.set_tuning(elem_threads_per_sm=threads, elem_persistent=persistent)

    def run(frozen=None):
        R = ws.ev.evaluate(phi, flow, frozen=frozen).clone()
        return R, ws.ev.rho_tilde.clone(), ws.ev.jacobian().to_scipy(), ws.ev.read_monitors()
    R, rt, J, mon = run()
    assert 0 < mon["n_supersonic"] < m.n_tets
    up, br = ws.freeze(phi, flow)
    live = torch.full_like(br, -1)
    Rl, rtl, Jl, monl = run((up, live))
    assert torch.equal(Rl, R) and torch.equal(rtl, rt) and monl == mon
    assert np.array_equal(Jl.data, J.data) and np.array_equal(Jl.indices, J.indices)
    part = torch.where(torch.arange(m.n_tets, device="cuda") % 3 == 0, br, live)
    for fz in ((up, br), (up, part)):
        Rf, rtf, Jf, _ = run(fz)   # (a frozen element of its own upstream counts no switch)
        assert rel_err(Rf.cpu().numpy(), R.cpu().numpy()) < REL_TOL
        assert rel_err(rtf.cpu().numpy(), rt.cpu().numpy()) < 1e-14
        assert sparse_rel_err(Jf, J) < REL_TOL
