"""Every form of the mixed kernels (scheme x kernel function x box, all compile-
time) against the FP64 form on one state, at an even and an odd size.

Sums of up to 200 positive FP32 terms, each of about 20 roundings, agree to
220 * 2^-24 < 2e-5; h follows the sums with slope 1/3 and Newton's own tolerance
is second order (1e-4 squared).  The force's terms have both signs: its error is
bounded by their magnitudes' sum, for a random cloud (neighbours N) about
sqrt(N) < 15 times the force, so 15 * 2e-5 and a factor 3 in the norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [600, 1001])
@pytest.mark.parametrize("periodic", [0, 1])
@pytest.mark.parametrize("kernel", ["CUBIC_SPLINE", "WENDLAND", "GAUSSIAN"])
@pytest.mark.parametrize("scheme", ["SSPH", "DISPH", "GSPH", "GDISPH"])
def test_mixed_against_fp64(gpu, scheme, kernel, periodic, n):
    r = np.random.default_rng(n)
    # a jittered lattice: no close pairs, smooth pressure
    m = int(np.ceil(n ** (1.0 / 3.0)))
    x = (np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] + 0.5) / m - 0.5
    x += r.uniform(-0.2, 0.2, x.shape) / m
    f = {f"pos_{a}": x[:, k] for k, a in enumerate("xyz")}
    for k, a in enumerate("xyz"):
        f[f"vel_{a}"] = 0.3 * np.sin(2 * np.pi * x[:, (k + 1) % 3])
    f["mass"] = np.full(n, 1.0 / m ** 3)
    f["ene"] = 1.5 + 0.5 * np.cos(2 * np.pi * x[:, 0])
    f["sound"] = np.sqrt(5.0 / 3.0 * (2.0 / 3.0) * f["ene"])
    f["alpha"], f["dens"] = np.ones(n), np.ones(n)   # (the first h follows from the density)
    out = {}
    for precision in (gpu.FP64, gpu.MIXED):
        p = gpu.config_params("shear_disph", sph_type=getattr(gpu, scheme), kernel=getattr(gpu, kernel),
                              periodic=periodic, range_min=(-0.5,) * 3, range_max=(0.5,) * 3, neighbor_number=50,
                              precision=precision)
        with gpu.Simulation(p) as sim:
            sim.upload(f)
            sim.initialize()
            out[precision] = sim.download(["sml", "dens", "pres", "acc_x", "acc_y", "acc_z", "neighbor"])
    a, b = out[gpu.FP64], out[gpu.MIXED]
    for k in ("sml", "dens", "pres"):
        np.testing.assert_allclose(b[k], a[k], rtol=2e-5, err_msg=k)
    d = np.stack([b[f"acc_{k}"] - a[f"acc_{k}"] for k in "xyz"])
    assert np.linalg.norm(d) < 3 * 15 * 2e-5 * np.linalg.norm(np.stack([a[f"acc_{k}"] for k in "xyz"]))
    assert np.max(np.abs(b["neighbor"] - a["neighbor"])) <= 1
