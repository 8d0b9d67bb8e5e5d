"""The weighted density's neighbour lists are on the device once, in the form
its sweep reads; the lists that a caller asks for come out of that form,
at every depth and after a change of depth."""

import numpy as np
import pytest

from conftest import has_cuda

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]


def test_lists_are_held_once():
    from up3d_b200 import _lib as L
    from up3d_b200.kernels.upwind import UpwindOperator
    from up3d_b200.mesh.device import DeviceMesh
    from up3d_b200.mesh.kuhn import kuhn_box
    nodes, elements = kuhn_box(40, 20, 20)
    dm = DeviceMesh(nodes, elements)
    before = L.pool_stats()["live_bytes"]
    upw = UpwindOperator(nodes, elements, weighted=True, mode="kernel", mesh=dm)
    built = L.pool_stats()["live_bytes"] - before
    total = upw._neighborhoods()[2]
    # the lists, 8 bytes an element of offsets, and padding below an eighth
    assert built < 4 * total * 1.125 + 8.5 * dm.n_tets + (8 << 20), (built, 4 * total)
    assert L.pool_stats()["live_bytes"] - before == built
    assert len(upw._nb_idx) == total       # asked for: a second copy


@pytest.mark.parametrize("shape", [(1, 1, 1), (5, 3, 2), (16, 5, 4)])
def test_exported_lists_at_each_depth(shape):
    from up3d_b200.kernels.upwind import UpwindOperator, build_upstream_neighborhoods
    from up3d_b200.mesh.device import DeviceMesh
    from up3d_b200.mesh.kuhn import bump_channel
    m = bump_channel(*shape, amplitude=0.05, seed=1)
    dm = DeviceMesh(m.nodes, m.elements)
    rng = np.random.default_rng(0)
    grad, q2 = rng.standard_normal((m.n_tets, 3)), rng.uniform(0.5, 2.0, m.n_tets)
    rho = rng.uniform(0.5, 1.0, m.n_tets)
    for depth in (3, 1, 5, 4, 2, 6):       # 5 and 6: built on the host
        upw = UpwindOperator(m.nodes, m.elements, weighted=True, mode="kernel", nbr_depth=depth, mesh=dm)
        rt = upw.rho_tilde(grad, q2, rho, 0.8, 1.5, 0.95).copy()
        off, idx = build_upstream_neighborhoods(upw.face_neighbors, depth)
        assert np.array_equal(upw._nb_off, off) and np.array_equal(upw._nb_idx, idx)
        assert np.array_equal(upw._nb_idx, idx)
        assert np.array_equal(upw.rho_tilde(grad, q2, rho, 0.8, 1.5, 0.95), rt)
