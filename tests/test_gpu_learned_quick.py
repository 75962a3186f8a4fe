"""The learned start's Newton steps by branch-free operations against the general
ones: pressures scaled by 2^k take the intermediates (up to the fourth power of a
wave speed) out of the short forms' range, and scale p* exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2_unit", [60, 100, 160, -60, -100, -160])
def test_star_states_scale_exactly(gpu, log2_unit):
    r = np.random.default_rng(5)
    n = 4099
    s = np.empty((n, 7))
    s[:, [1, 4]] = np.exp(r.uniform(-3, 3, (n, 2)))
    s[:, [2, 5]] = np.exp(r.uniform(-4, 4, (n, 2)))
    s[:, [0, 3]] = r.uniform(-1, 1, (n, 2))
    s[:, 6] = 1.4
    t = s.copy()
    # p and rho by 2^(2 k): velocities stay, wave speeds scale by 2^(2 k)
    t[:, [1, 2, 4, 5]] *= 2.0 ** (2 * log2_unit)
    with gpu.Simulation(gpu.config_params("tube_gsph")) as sim:
        sim.load_riemann_mlp()
        p0, v0, it0, fb0 = sim.riemann_batch(s, mode=1)
        p1, v1, it1, fb1 = sim.riemann_batch(t, mode=1)
    # the floor 1e-25 of p is no power of the unit
    ok = (p0 > 1e-20) & (p1 > 1e-20)
    assert ok.sum() > (0.9 * n if log2_unit > 0 else -1)
    np.testing.assert_array_equal(p1[ok], p0[ok] * 2.0 ** (2 * log2_unit))
    np.testing.assert_array_equal(v1[ok], v0[ok])
    np.testing.assert_array_equal(it1[ok], it0[ok])
