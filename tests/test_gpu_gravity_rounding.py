"""The gravity walk's correctly rounded quotients and roots (csrc/rounded.cuh)
against the oracle's IEEE operations: every acceleration and potential bit for
bit.  Units from where the short forms hold to where only the general
operations do (2^-80 .. 2^80 in h and r^2, 2^-300 .. 2^300 in d^2), smoothing
lengths that put pairs on every branch of the softening, open and periodic
boxes, and both register budgets of the kernel (the larger sphere)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(n, scale, seed):
    r = np.random.default_rng(seed)
    f = {f"pos_{a}": scale * r.uniform(-0.5, 0.5, n) for a in "xyz"}
    f["mass"] = r.uniform(0.5, 2.0, n) / n
    f["sml"] = scale * np.exp(r.uniform(np.log(0.01), np.log(0.6), n))
    for a in "xyz":
        f[f"acc_{a}"] = r.standard_normal(n) / scale
    return f


def _compare(gpu, O, p, f):
    o = O.Oracle(p, f)
    o.tree_make()
    o.gravity_force()
    ref = o.download()
    with gpu.Simulation(p) as sim:
        sim.upload(f)
        sim.tree_make()
        sim.gravity_force()
        out = sim.download(["acc_x", "acc_y", "acc_z", "phi"])
    for k in out:
        np.testing.assert_array_equal(out[k], ref[k], err_msg=k)


@pytest.mark.parametrize("periodic", [0, 1])
@pytest.mark.parametrize("log2_unit", [0, 39, -42, 100, -100, 160, -160])
def test_gravity_bitexact_in_any_unit(gpu, O, log2_unit, periodic):
    unit = 2.0 ** log2_unit
    p = gpu.config_params("evrard_ssph", periodic=periodic, range_min=(-0.5 * unit,) * 3,
                          range_max=(0.5 * unit,) * 3)
    _compare(gpu, O, p, _cloud(3001, unit, 7))


@pytest.mark.parametrize("n", [1, 2, 31, 33, 148 * 16 * 32 * 4 + 17])
def test_gravity_bitexact_sizes(gpu, O, n):
    f = _cloud(n, 1.0, n)
    f["sml"] = np.minimum(f["sml"], 3.0 / n ** (1.0 / 3.0))
    _compare(gpu, O, gpu.config_params("evrard_ssph"), f)
