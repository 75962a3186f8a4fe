"""PreInteraction's masked candidates (FP64 form): a particle whose mass is NaN
or infinite touches the sums of those whose kernel it lies in and of no others
(a masked candidate adds zeros).  Against the oracle, over the lists of 1.2 times
the guess in which the smoothing length is searched: densities and smoothing
lengths that are no numbers in the same places."""
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


@pytest.mark.parametrize("periodic", [0, 1])
@pytest.mark.parametrize("kernel", ["CUBIC_SPLINE", "WENDLAND", "GAUSSIAN"])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("kind", ["SSPH", "DISPH", "GSPH", "GDISPH"])
def test_bad_mass_stays_in_its_kernels(gpu, O, kind, value, kernel, periodic):
    n = 600
    p = gpu.default_params(sph_type=getattr(gpu, kind), kernel=getattr(gpu, kernel), neighbor_number=30, gamma=1.4,
                           iterative_sml=1, periodic=periodic, range_min=(-0.5,) * 3, range_max=(0.5,) * 3)
    f = _state(n, 2)
    f["mass"][17] = value
    o = O.Oracle(p, f)
    o.tree_make()
    o.pre_interaction()
    ref = o.download(["dens", "sml"])
    with gpu.Simulation(p) as sim:
        sim.upload(f)
        sim.tree_make()
        sim.pre_interaction()
        out = sim.download(["dens", "sml"])
    others = np.arange(n) != 17
    bad = np.sum(~np.isfinite(ref["dens"][others]) | ~np.isfinite(ref["sml"][others]))
    assert bad < n // 2 and (bad > 0 or value == np.inf)
    for k in ("dens", "sml"):
        np.testing.assert_array_equal(np.isfinite(out[k][others]), np.isfinite(ref[k][others]), err_msg=k)
