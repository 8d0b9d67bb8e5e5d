"""The streamline-kernel density where only some neighbourhoods reach the
critical Mach number (the others keep their own density without forming the
weights): scattered supercritical elements, speeds at the critical one, and
past the vacuum limit, against the oracle."""

import numpy as np
import pytest

from conftest import REL_TOL, has_cuda, rel_err

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]

M_INF, C, M_CRIT, GAMMA = 0.8, 1.5, 0.95, 1.4


def _critical_q2(m):
    return m * m * (1.0 + 0.2 * M_INF ** 2) / (M_INF ** 2 * (1.0 + 0.2 * m * m))


@pytest.mark.parametrize("shape", [(1, 1, 1), (7, 5, 3), (16, 4, 5)])
@pytest.mark.parametrize("depth", [1, 3])
@pytest.mark.parametrize("kind", ["none", "scattered", "critical", "vacuum"])
def test_scattered_supercritical_elements(shape, depth, kind):
    from oracle import oracle as O
    from up3d_b200.kernels.upwind import UpwindOperator
    from up3d_b200.mesh.kuhn import bump_channel
    m = bump_channel(*shape, amplitude=0.05, seed=1)
    rng = np.random.default_rng(shape[0] + depth)
    grad, _ = O.PicardOperator(m.nodes, m.elements).velocities(
        m.nodes[:, 0] + 0.05 * rng.standard_normal(len(m.nodes)))
    q2 = rng.uniform(0.6, 0.95, m.n_tets) * _critical_q2(M_CRIT)
    some = rng.choice(m.n_tets, size=max(1, m.n_tets // 60), replace=False)
    if kind == "scattered":
        q2[some] = _critical_q2(1.2)
    elif kind == "critical":
        q2[some] = _critical_q2(M_CRIT) * (1.0 + rng.choice([-1e-14, 0.0, 1e-14], size=len(some)))
    elif kind == "vacuum":
        q2[some] = 1.05 * (1.0 + 1.0 / (0.2 * M_INF ** 2))
    rho = rng.uniform(0.5, 1.0, m.n_tets)
    ref = O.UpwindOperator(m.nodes, m.elements, weighted=True, mode="kernel", nbr_depth=depth)
    upw = UpwindOperator(m.nodes, m.elements, weighted=True, mode="kernel", nbr_depth=depth)
    r = ref.rho_tilde(grad, q2, rho, M_INF, C, M_CRIT).copy()
    d = upw.rho_tilde(grad, q2, rho, M_INF, C, M_CRIT)
    assert rel_err(d, r) < REL_TOL
    assert np.abs(np.asarray(upw.nu) - ref.nu).max() < REL_TOL
    if kind in ("none", "scattered"):
        assert upw.n_supersonic == ref.n_supersonic
        assert (upw.n_supersonic > 0) == (kind == "scattered")
