"""The group walk in thin periodic boxes against the per-lane walk (which runs
the reference's tests one by one): equal sets where the box is a little longer
than two radii (a pair's nearest image may differ between the lanes of a
group), shorter than that, and for particles whose octree order jumps inside a
warp's window, for both searches and at sizes around a warp and a block."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sets(off, ids):
    return [np.sort(ids[off[i]:off[i + 1]]) for i in range(len(off) - 1)]


@pytest.mark.parametrize("is_ij", [False, True])
@pytest.mark.parametrize("n", [33, 64, 1500])
@pytest.mark.parametrize("thin", [1.5, 1.98, 2.01, 2.05, 2.5, 4.0])
def test_group_walk_equals_per_lane_walk(gpu, thin, n, is_ij):
    h = 0.04
    box = np.array([1.0, thin * h, thin * h])
    r = np.random.default_rng(int(100 * thin) + n)
    x = r.uniform(size=(n, 3)) * box
    x[: n // 3, 0] = 0.001 * r.uniform(size=n // 3)       # a dense slab: runs and jumps in one window
    p = gpu.config_params("tube_gsph", range_min=(0.0, 0.0, 0.0), range_max=tuple(box))
    f = {"pos_x": x[:, 0].copy(), "pos_y": x[:, 1].copy(), "pos_z": x[:, 2].copy(), "mass": np.full(n, 1.0 / n),
         "sml": h * r.uniform(0.2, 1.0, n)}
    out = []
    with gpu.Simulation(p) as sim:
        sim.upload(f)
        sim.tree_make()
        sim.set_kernel()
        for mode in (0, 1):
            sim.set_walk_mode(mode)
            out.append(_sets(*sim.neighbor_search(is_ij)))
        assert sim.counters()["walk_fallbacks"] == 0
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
