"""The mixed gravity walk's two kinds of leaf: one particle, named by the node's
own record, and several, whose range is read from the tree.  With a vanishing
opening angle every leaf is opened and the walk is the direct sum, so the FP64
form gives the same sum of the same pairs.

The bound: a pair's term takes at most 8 FP32 roundings (2^-24 each) on a
polynomial whose terms' magnitudes sum to at most 150 times the result (at
u = 2), so the difference is below 150 * 8 * 2^-24 of the sum of the terms'
magnitudes; a leaf's particle lost or counted twice is 1/n of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 33, 700])
@pytest.mark.parametrize("leaf_particle_num", [1, 2, 8])
def test_mixed_leaves_direct_sum(gpu, n, leaf_particle_num):
    r = np.random.default_rng(n)
    f = {f"pos_{a}": r.uniform(-0.5, 0.5, n) for a in "xyz"}
    f["mass"] = np.full(n, 1.0 / n)
    f["sml"] = np.exp(r.uniform(np.log(0.01), np.log(0.6), n))
    out = {}
    for precision in (gpu.FP64, gpu.MIXED):
        p = gpu.config_params("evrard_ssph", precision=precision, theta=1e-6,
                              leaf_particle_num=leaf_particle_num)
        with gpu.Simulation(p) as sim:
            sim.upload(f)
            sim.tree_make()
            sim.gravity_force()
            out[precision] = sim.download(["acc_x", "acc_y", "acc_z", "phi", "mass"])
    acc = np.stack([out[gpu.FP64][f"acc_{a}"] for a in "xyz"], 1)
    d = np.stack([out[gpu.MIXED][f"acc_{a}"] for a in "xyz"], 1) - acc
    # the magnitudes' sum, from above: softening only weakens a pair
    x = np.stack([f[f"pos_{a}"] for a in "xyz"], 1)
    r2 = ((x[:, None] - x[None]) ** 2).sum(2)
    np.fill_diagonal(r2, np.inf)
    mag = (f["mass"][None] / r2).sum(1)
    bound = 150 * 8 * 2.0 ** -24
    assert np.all(np.abs(d).max(1) <= bound * mag)
    phi = np.abs(out[gpu.MIXED]["phi"] - out[gpu.FP64]["phi"])
    assert np.all(phi <= bound * (f["mass"][None] / np.sqrt(r2)).sum(1))
