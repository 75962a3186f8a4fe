"""Two particles that approach each other at distances whose square leaves the
range of the short forms (r^2 below 2^-1000): the signal velocity, and with it
the time step, are the oracle's finite ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dist", [1e-120, 1e-150, 1e-152, 1e-155, 1e-160])
@pytest.mark.parametrize("kernel", ["CUBIC_SPLINE", "WENDLAND", "GAUSSIAN"])
@pytest.mark.parametrize("kind", ["SSPH", "DISPH", "GSPH", "GDISPH"])
def test_signal_velocity_of_a_close_pair(gpu, O, kind, kernel, dist):
    n = 600
    r = np.random.default_rng(3)
    f = {f"pos_{a}": r.uniform(-0.5, 0.5, n) for a in "xyz"}
    f.update({f"vel_{a}": r.standard_normal(n) for a in "xyz"})
    f["mass"] = r.uniform(0.5, 2.0, n) / n
    f["dens"] = r.uniform(0.5, 2.0, n)
    f["ene"] = np.exp(r.uniform(-2, 2, n))
    f["pres"] = 0.4 * f["dens"] * f["ene"]
    f["sound"] = np.sqrt(1.4 * f["pres"] / f["dens"])
    f["alpha"] = r.uniform(0.1, 2.0, n)
    for a in "xyz":
        f[f"pos_{a}"][5] = f[f"pos_{a}"][6] = 0.0
    f["pos_x"][6] = dist
    f["vel_x"][5], f["vel_x"][6] = 20.0, -20.0    # the fastest pair: it sets min h / v_sig
    p = gpu.default_params(sph_type=getattr(gpu, kind), kernel=getattr(gpu, kernel), neighbor_number=30, gamma=1.4,
                           iterative_sml=0, leaf_particle_num=2)
    o = O.Oracle(p, f)
    o.tree_make()
    o.pre_interaction()
    with gpu.Simulation(p) as sim:
        sim.upload(f)
        sim.tree_make()
        sim.pre_interaction()
        hvs = sim.h_per_v_sig()
    assert o.h_per_v_sig() > 0.0
    # r from a subnormal r^2 keeps 2^-(1074 + log2 r^2) of its bits: 2^-12 at 1e-160
    np.testing.assert_allclose(hvs, o.h_per_v_sig(), rtol=1e-3 if dist < 1e-154 else 1e-12)
