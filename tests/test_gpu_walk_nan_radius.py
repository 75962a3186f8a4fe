"""A particle whose radius is NaN has an empty list in either search, as in the
per-lane walk (r^2 < NaN holds for no pair, with whatever kernel size a node
has: src/bhtree.cpp:277-316), and the others' lists are untouched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("is_ij", [False, True])
@pytest.mark.parametrize("periodic", [0, 1])
def test_nan_radius_finds_nothing(gpu, periodic, is_ij):
    n = 600
    r = np.random.default_rng(6)
    p = gpu.config_params("blast_gsph", periodic=periodic)
    f = {f"pos_{a}": r.uniform(-0.5, 0.5, n) for a in "xyz"}
    f["mass"], f["sml"] = np.full(n, 1.0 / n), r.uniform(0.1, 0.2, n)
    f["sml"][[17, 300, 301]] = np.nan
    out = []
    with gpu.Simulation(p) as sim:
        sim.upload(f)
        sim.tree_make()
        sim.set_kernel()
        for mode in (0, 1):
            sim.set_walk_mode(mode)
            off, ids = sim.neighbor_search(is_ij)
            out.append([np.sort(ids[off[i]:off[i + 1]]) for i in range(n)])
    assert all(len(out[1][i]) == 0 for i in (17, 300, 301))
    for i in range(n):
        np.testing.assert_array_equal(out[0][i], out[1][i], err_msg=f"particle {i}")
