"""Evaluators and operators that share one mesh handle, whose workspace holds
the Term-3 entries outside the P1 pattern of the last Jacobian formed on it:
merging an earlier one is refused, and a merge never writes past the arrays
it is given."""

import ctypes

import numpy as np
import pytest

from conftest import has_cuda

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]


def _two_evaluators():
    import torch
    from up3d_b200.mesh.device import DeviceMesh
    from up3d_b200.mesh.kuhn import bump_channel, pocket_state
    from up3d_b200.solve.fused import FlowParams, ResidualJacobian
    mesh = bump_channel(20, 6, 5, amplitude=0.08, seed=5)
    dm = DeviceMesh(mesh.nodes, mesh.elements)
    state = [torch.from_numpy(pocket_state(mesh, f)).cuda() for f in ("mixed", "accelerating")]
    a, b = ResidualJacobian(dm), ResidualJacobian(dm)
    flow = FlowParams(m_inf=0.8)
    extras = []
    for ev, phi in zip((a, b), state):
        ev.evaluate(phi, flow)
        extras.append(ev.read_monitors()["n_term3_extra"])
    if extras[0] > extras[1]:       # a: fewer extras than b
        a, b, state, extras = b, a, state[::-1], extras[::-1]
    assert 0 < extras[0] < extras[1]
    return mesh, dm, flow, state, a, b


@pytest.mark.parametrize("between", ["evaluator", "operator"])
def test_merge_of_an_earlier_jacobian_is_refused(between):
    mesh, dm, flow, state, a, b = _two_evaluators()
    a.evaluate(state[0], flow)
    own = a.jacobian().to_scipy()
    a.evaluate(state[0], flow)
    if between == "evaluator":
        b.evaluate(state[1], flow)
        assert b.jacobian().nnz > own.nnz
    else:
        import torch
        from up3d_b200.kernels.jacobian import PicardOperator
        op = PicardOperator(mesh.nodes, mesh.elements, mesh=dm)
        one = torch.ones(dm.n_tets, dtype=torch.float64, device="cuda")
        up = torch.arange(dm.n_tets, device="cuda").roll(dm.n_tets // 2)   # far: all outside the pattern
        J = op.assemble_newton_jacobian(state[1], one, -one, -one, up)
        assert J.nnz > own.nnz
    with pytest.raises(RuntimeError, match="evaluate again"):
        a.jacobian()
    # a residual without a Jacobian leaves the extras alone
    a.evaluate(state[0], flow)
    b.evaluate(state[1], flow, jacobian=False)
    again = a.jacobian().to_scipy()
    assert np.array_equal(again.indptr, own.indptr) and np.array_equal(again.indices, own.indices)
    assert np.array_equal(again.data, own.data)


@pytest.mark.parametrize("short", [0, 1, 7, 1000])
def test_merge_stays_within_its_capacity(short):
    import torch
    from up3d_b200 import _lib as L
    _, dm, flow, state, a, _ = _two_evaluators()
    a.evaluate(state[0], flow)
    J = a.jacobian()
    total, room = J.nnz, 64
    indptr = torch.empty(dm.n_nodes + 1, dtype=torch.int32, device="cuda")
    indices = torch.full((total + room,), -7, dtype=torch.int32, device="cuda")
    data = torch.full((total + room,), -7.0, dtype=torch.float64, device="cuda")
    nnz = ctypes.c_int64()

    def merge():
        L.call("up3d_jacobian_merge", dm.handle, a.data.data_ptr(), indptr.data_ptr(), indices.data_ptr(),
               data.data_ptr(), total - short, -1, ctypes.byref(nnz), L.stream_ptr())
    if short:
        with pytest.raises(ValueError, match="more entries"):
            merge()
    else:
        merge()
    assert nnz.value == total
    assert bool((indices[total - short:] == -7).all()) and bool((data[total - short:] == -7.0).all())
    assert torch.equal(data[:total - short], J.data[:total - short])
    assert torch.equal(indices[:total - short], J.indices[:total - short])
