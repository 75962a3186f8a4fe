"""A slope that is not a number, or infinite against a zero difference, in the
second-order Riemann states of the FP64 form: FluidForce's outputs are NaN
exactly where the oracle's are.  (gsph's iterative solver floors a NaN
pressure, so its accelerations stay finite there and du/dt does not.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OUT = ["acc_x", "acc_y", "acc_z", "dene"]


def _state(n, seed):
    r = np.random.default_rng(seed)
    f = {f"pos_{a}": r.uniform(-0.5, 0.5, n) for a in "xyz"}
    f.update({f"vel_{a}": r.standard_normal(n) for a in "xyz"})
    f["mass"] = r.uniform(0.5, 2.0, n) / n
    f["dens"] = r.uniform(0.5, 2.0, n)
    f["ene"] = np.exp(r.uniform(-2, 2, n))
    f["pres"] = 0.4 * f["dens"] * f["ene"]
    f["sound"] = np.sqrt(1.4 * f["pres"] / f["dens"])
    f["sml"] = r.uniform(0.8, 1.4, n) * (30.0 / n) ** (1.0 / 3.0) * 0.62
    f["alpha"], f["balsara"] = r.uniform(0.1, 2.0, n), r.uniform(0, 1, n)
    f["gradh"] = 1e-4 * r.uniform(0.5, 1.5, n)
    for g in ("d", "p", "v0", "v1", "v2"):
        for a in "xyz":
            f[f"grad_{g}_{a}"] = 0.1 * r.standard_normal(n)
    return f


@pytest.mark.parametrize("field", ["grad_d_x", "grad_p_y", "grad_v1_z"])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("form", ["gsph", "gsph_hll", "gdisph"])
def test_nan_slope_reaches_the_outputs(gpu, O, form, value, field):
    n = 600
    p = gpu.default_params(sph_type=gpu.GDISPH if form == "gdisph" else gpu.GSPH, gamma=1.4, neighbor_number=30,
                           riemann_solver=gpu.RIEMANN_HLL if form == "gsph_hll" else gpu.RIEMANN_ITERATIVE,
                           gsph_2nd_order=1, use_ac=1)
    f = _state(n, 2)
    f[field][17] = value
    if value == np.inf:
        # the infinite slope meets differences of exactly zero
        for k in ("vel_x", "vel_y", "vel_z", "dens", "pres", "ene", "sound"):
            f[k][:] = f[k][0]
    o = O.Oracle(p, f)
    o.tree_make()
    o.set_kernel()
    o.set_dt(0.01)
    o.fluid_force()
    ref = o.download(OUT)
    with gpu.Simulation(p) as sim:
        sim.upload(f)
        sim.tree_make()
        sim.set_kernel()
        sim.set_dt(0.01)
        sim.fluid_force()
        out = sim.download(OUT)
    bad = sum(int(np.isnan(ref[k]).sum()) for k in OUT)
    assert 0 < bad < 4 * n
    for k in OUT:
        np.testing.assert_array_equal(np.isnan(out[k]), np.isnan(ref[k]), err_msg=k)
