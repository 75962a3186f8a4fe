"""The general operations (csrc/rounded.cuh, Ieee) behind FluidForce's branch-free
ones, in the forms and at the units where they are the ones that run.

Forces: masses, densities and pressures times 2^+-410 take 1 / (rho_i + rho_j)
(ssph, disph, gdisph), P_j / rho_j^2 and HLL's 1 / (c_1 - c_2) past 2^+-400, where
each pair is computed again; accelerations and du/dt do not change, and every
product stays finite.  Against the oracle in the plain unit: the products around
the two kinds of operations are fused differently, so bits may differ.  Learned
start: pressures and densities times 2^(2 k), k over 200, take each Newton step's
quotients past 2^400 (its largest products are 2^(4 k)); p* scales exactly."""
import numpy as np
import pytest

from test_gpu_force_quick import _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [0, 1])
@pytest.mark.parametrize("kernel", ["CUBIC_SPLINE", "WENDLAND", "GAUSSIAN"])
@pytest.mark.parametrize("log2_scale", [410, -410])
@pytest.mark.parametrize("form", ["ssph", "disph", "gdisph", "gsph_hll"])
def test_force_by_general_operations(gpu, O, form, log2_scale, kernel, periodic):
    kind = form.split("_")[0]
    p = gpu.default_params(sph_type=getattr(gpu, kind.upper()), kernel=getattr(gpu, kernel), use_ac=1, gamma=1.4,
                           use_time_dependent_av=1, periodic=periodic, range_min=(-0.5,) * 3, range_max=(0.5,) * 3,
                           riemann_solver=gpu.RIEMANN_HLL, gsph_2nd_order=1)
    f = _state(1000, periodic, 3)
    if kind in ("disph", "gdisph"):
        f["gradh"] = f["gradh"] * 1e-4
    o = O.Oracle(p, f)
    o.tree_make()
    o.set_kernel()
    o.set_dt(0.01)
    o.fluid_force()
    ref = o.download(["acc_x", "acc_y", "acc_z", "dene"])
    scale = 2.0 ** log2_scale
    q = dict(f)
    names = ["mass", "dens", "pres"] + [f"grad_{g}_{a}" for g in "dp" for a in "xyz"]
    for k in names + (["gradh"] if kind in ("disph", "gdisph") else []):
        q[k] = q[k] * scale
    p.alpha_ac = 1.0 / scale       # the conductivity term carries a mass
    with gpu.Simulation(p) as sim:
        sim.upload(q)
        sim.tree_make()
        sim.set_kernel()
        sim.set_dt(0.01)
        sim.fluid_force()
        out = sim.download(["acc_x", "acc_y", "acc_z", "dene"])
    # some 40 roundings of 2^-53 in each of up to 100 terms, which add up to some
    # 30 times the largest sum: 1.3e-13 of it
    for k in ref:
        scale_k = np.max(np.abs(ref[k]))
        assert np.all(np.isfinite(out[k])) and scale_k > 0.0
        np.testing.assert_allclose(out[k], ref[k], rtol=0.0, atol=1e-12 * scale_k, err_msg=k)


@pytest.mark.parametrize("log2_unit", [205, 215, 225])
def test_learned_start_by_general_operations(gpu, log2_unit):
    r = np.random.default_rng(5)
    n = 4099
    s = np.empty((n, 7))
    s[:, [1, 4]] = np.exp(r.uniform(-3, 3, (n, 2)))
    s[:, [2, 5]] = np.exp(r.uniform(-4, 4, (n, 2)))
    s[:, [0, 3]] = r.uniform(-1, 1, (n, 2))
    s[:, 6] = 1.4
    t = s.copy()
    t[:, [1, 2, 4, 5]] *= 2.0 ** (2 * log2_unit)
    with gpu.Simulation(gpu.config_params("tube_gsph")) as sim:
        sim.load_riemann_mlp()
        p0, v0, it0, fb0 = sim.riemann_batch(s, mode=1)
        p1, v1, it1, fb1 = sim.riemann_batch(t, mode=1)
    ok = p0 > 1e-20     # (the floor 1e-25 of p is no power of the unit)
    assert ok.sum() > 0.9 * n and np.all(np.isfinite(p1))
    np.testing.assert_array_equal(p1[ok], p0[ok] * 2.0 ** (2 * log2_unit))
    np.testing.assert_array_equal(v1[ok], v0[ok])
    np.testing.assert_array_equal(it1[ok], it0[ok])
    np.testing.assert_array_equal(fb1[ok], fb0[ok])
