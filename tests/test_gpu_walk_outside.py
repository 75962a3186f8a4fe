"""The group walk with particles outside the periodic box: a pair's nearest image
is taken once (include/periodic.hpp:34-72), so an offset of two boxes stays one
box long.  The lists of the particles inside the box equal the per-lane walk's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sets(off, ids):
    return [np.sort(ids[off[i]:off[i + 1]]) for i in range(len(off) - 1)]


@pytest.mark.parametrize("is_ij", [False, True])
@pytest.mark.parametrize("wide", [0.15, 0.45])
@pytest.mark.parametrize("shift", [2.0, -2.0, 3.0, -4.0])
def test_group_walk_takes_one_image(gpu, shift, wide, is_ij):
    n, nout = 600, 40
    r = np.random.default_rng(6)
    x = r.uniform(-0.5, 0.5, (n, 3))
    x[:nout, 0] += shift
    p = gpu.config_params("blast_gsph")
    f = {f"pos_{a}": x[:, k].copy() for k, a in enumerate("xyz")}
    f["mass"], f["sml"] = np.full(n, 1.0 / n), wide * r.uniform(0.6, 1.0, n)
    out = []
    with gpu.Simulation(p) as sim:
        sim.upload(f)
        sim.tree_make()
        sim.set_kernel()
        for mode in (0, 1):
            sim.set_walk_mode(mode)
            out.append(_sets(*sim.neighbor_search(is_ij)))
    for i in range(nout, n):
        np.testing.assert_array_equal(out[0][i], out[1][i], err_msg=f"particle {i}")
