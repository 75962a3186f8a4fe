"""FluidForce's branch-free quotients and roots (csrc/rounded.cuh, Quick) against
its general operations (Ieee), pair by pair through the sums: with all masses
scaled by 2^210 (densities, pressures and, for disph and gdisph, the grad-h
terms with them, the conductivity's coefficient inversely) the accelerations and du/dt are the same numbers, but 1 / rho^2
leaves the range of the quick forms, so every pair takes the general ones.  The
results must be equal bit for bit.  (Scaled up only: the Riemann solver floors
its pressure at 1e-25.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(n, periodic, seed):
    r = np.random.default_rng(seed)
    f = {f"pos_{a}": r.uniform(-0.5, 0.5, n) for a in "xyz"}
    f.update({f"vel_{a}": r.standard_normal(n) for a in "xyz"})
    f["mass"] = r.uniform(0.5, 2.0, n) / n
    f["dens"] = r.uniform(0.3, 3.0, n)
    f["ene"] = np.exp(r.uniform(-3, 3, n))
    f["pres"] = 0.4 * f["dens"] * f["ene"]
    f["sound"] = np.sqrt(1.4 * f["pres"] / f["dens"])
    f["sml"] = r.uniform(0.5, 1.5, n) * (20.0 / n) ** (1.0 / 3.0) * 0.62
    f["alpha"], f["balsara"] = r.uniform(0.1, 2.0, n), r.uniform(0, 1, n)
    f["gradh"] = r.uniform(0.5, 1.5, n)
    for g in ("d", "p", "v0", "v1", "v2"):
        for a in "xyz":
            f[f"grad_{g}_{a}"] = r.standard_normal(n)
    return f


@pytest.mark.parametrize("periodic", [0, 1])
@pytest.mark.parametrize("kernel", ["CUBIC_SPLINE", "WENDLAND", "GAUSSIAN"])
@pytest.mark.parametrize("form", ["ssph", "disph", "gdisph", "gsph", "gsph_hll", "gsph_first"])
def test_quick_equals_general_operations(gpu, form, kernel, periodic):
    kind = form.split("_")[0]
    p = gpu.default_params(sph_type=getattr(gpu, kind.upper()), kernel=getattr(gpu, kernel), use_ac=1, gamma=1.4,
                           use_time_dependent_av=1, periodic=periodic, range_min=(-0.5,) * 3, range_max=(0.5,) * 3,
                           riemann_solver=gpu.RIEMANN_HLL if form == "gsph_hll" else gpu.RIEMANN_ITERATIVE,
                           gsph_2nd_order=0 if form == "gsph_first" else 1)
    f = _state(1000, periodic, 3)
    if kind in ("disph", "gdisph"):
        f["gradh"] = f["gradh"] * 1e-4
    out = []
    for scale in (1.0, 2.0 ** 210):
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
            out.append(sim.download(["acc_x", "acc_y", "acc_z", "dene"]))
    for k in out[0]:
        assert np.all(np.isfinite(out[0][k])) and np.any(out[0][k] != 0.0)
        np.testing.assert_array_equal(out[0][k], out[1][k], err_msg=k)
