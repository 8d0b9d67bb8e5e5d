"""The streamline-kernel density at speeds and densities that are NaN or
infinite: a neighbourhood with one takes the full sum, as if nothing were
skipped, against the oracle."""

import numpy as np
import pytest

from conftest import has_cuda

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]


@pytest.mark.parametrize("what", ["q2", "rho"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("speed", [0.6, 1.6])
def test_one_value_not_finite(what, value, speed):
    from oracle import oracle as O
    from up3d_b200.kernels.upwind import UpwindOperator
    from up3d_b200.mesh.kuhn import bump_channel
    m = bump_channel(9, 4, 5, amplitude=0.05, seed=1)
    rng = np.random.default_rng(3)
    grad, _ = O.PicardOperator(m.nodes, m.elements).velocities(
        m.nodes[:, 0] + 0.05 * rng.standard_normal(len(m.nodes)))
    q2 = rng.uniform(0.8, 1.0, m.n_tets) * speed
    rho = rng.uniform(0.5, 1.0, m.n_tets)
    (q2 if what == "q2" else rho)[[3, m.n_tets // 2]] = value
    ref = O.UpwindOperator(m.nodes, m.elements, weighted=True, mode="kernel")
    upw = UpwindOperator(m.nodes, m.elements, weighted=True, mode="kernel")
    r = ref.rho_tilde(grad, q2, rho, 0.8, 1.5, 0.95).copy()
    d = np.asarray(upw.rho_tilde(grad, q2, rho, 0.8, 1.5, 0.95))
    assert np.array_equal(np.isnan(d), np.isnan(r)) and np.array_equal(np.isnan(upw.nu), np.isnan(ref.nu))
    ok = np.isfinite(r)
    assert np.array_equal(d[~ok & ~np.isnan(r)], r[~ok & ~np.isnan(r)])
    np.testing.assert_allclose(d[ok], r[ok], rtol=1e-12)
    nu = np.isfinite(ref.nu)
    np.testing.assert_allclose(np.asarray(upw.nu)[nu], ref.nu[nu], rtol=1e-12, atol=1e-12)
