"""PreInteraction (FP64 form) of a particle that has no pairs because its
smoothing length is zero or NaN (a mass of zero, a negative one or a density
guess below zero): density and pressure are the oracle's, an empty sum, and so
are everyone else's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(n, seed):
    r = np.random.default_rng(seed)
    f = {f"pos_{a}": r.uniform(-0.5, 0.5, n) for a in "xyz"}
    f.update({f"vel_{a}": r.standard_normal(n) for a in "xyz"})
    f["mass"] = r.uniform(0.5, 2.0, n) / n
    f["dens"] = r.uniform(0.5, 2.0, n)
    f["ene"] = np.exp(r.uniform(-2, 2, n))
    f["pres"] = 0.4 * f["dens"] * f["ene"]
    f["sound"] = np.sqrt(1.4 * f["pres"] / f["dens"])
    f["alpha"] = r.uniform(0.1, 2.0, n)
    return f


@pytest.mark.parametrize("iterative", [0, 1])
@pytest.mark.parametrize("kernel", ["CUBIC_SPLINE", "WENDLAND", "GAUSSIAN"])
@pytest.mark.parametrize("field,value", [("mass", 0.0), ("mass", -1.0 / 600), ("dens", -1.0)])
@pytest.mark.parametrize("kind", ["SSPH", "DISPH", "GSPH", "GDISPH"])
def test_empty_sum_is_zero(gpu, O, kind, field, value, kernel, iterative):
    n = 600
    p = gpu.default_params(sph_type=getattr(gpu, kind), kernel=getattr(gpu, kernel), neighbor_number=30, gamma=1.4,
                           iterative_sml=iterative)
    f = _state(n, 2)
    f[field][17] = value
    o = O.Oracle(p, f)
    o.tree_make()
    o.pre_interaction()
    ref = o.download(["dens", "pres"])
    with gpu.Simulation(p) as sim:
        sim.upload(f)
        sim.tree_make()
        sim.pre_interaction()
        out = sim.download(["dens", "pres"])
    assert ref["dens"][17] == 0.0
    for k in ("dens", "pres"):
        np.testing.assert_array_equal(np.isnan(out[k]), np.isnan(ref[k]), err_msg=k)
        ok = np.isfinite(ref[k])
        # (a Newton step more or less at its 1e-4 bound moves h by 1e-8)
        np.testing.assert_allclose(out[k][ok], ref[k][ok], rtol=1e-7, err_msg=k)


@pytest.mark.parametrize("kind", ["SSPH", "DISPH", "GDISPH"])
def test_tiny_kernel_overflows_as_before(gpu, O, kind):
    """A neighbour of 1e200 masses leaves smoothing lengths whose kernel gradient
    overflows: 0 times it is NaN in the reference, though the sum is zero."""
    p = gpu.default_params(sph_type=getattr(gpu, kind), kernel=gpu.WENDLAND, neighbor_number=30, gamma=1.4)
    f = _state(600, 2)
    f["mass"][17] = 1e200
    o = O.Oracle(p, f)
    o.tree_make()
    o.pre_interaction()
    ref = o.download(["dens", "balsara"])
    with gpu.Simulation(p) as sim:
        sim.upload(f)
        sim.tree_make()
        sim.pre_interaction()
        out = sim.download(["dens", "balsara"])
    for k in ref:
        np.testing.assert_array_equal(np.isnan(out[k]), np.isnan(ref[k]), err_msg=k)
