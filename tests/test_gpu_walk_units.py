"""The group walk's FP32 classification in any unit of length: positions, radii
and box scaled by 2^k give the lists of the unscaled set (every other operation
of the walk scales exactly), also where offsets, their squares or both leave
FP32's range, with radii from far below the spacing to infinite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sets(off, ids):
    return [np.sort(ids[off[i]:off[i + 1]]) for i in range(len(off) - 1)]


def _lists(gpu, x, h, box, periodic, unit, is_ij, mode):
    p = gpu.config_params("tube_gsph", periodic=periodic, range_min=(0.0, 0.0, 0.0), range_max=tuple(box * unit))
    n = len(x)
    f = {f"pos_{a}": (x[:, k] * unit).copy() for k, a in enumerate("xyz")}
    f["mass"], f["sml"] = np.full(n, 1.0 / n), h * unit
    with gpu.Simulation(p) as sim:
        sim.upload(f)
        sim.tree_make()
        sim.set_kernel()
        sim.set_walk_mode(mode)
        out = _sets(*sim.neighbor_search(is_ij))
        assert sim.counters()["walk_fallbacks"] == 0
    return out


@pytest.mark.parametrize("is_ij", [False, True])
@pytest.mark.parametrize("periodic", [0, 1])
@pytest.mark.parametrize("odd", ["", "wide", "infinite", "small"])
def test_lists_do_not_depend_on_the_unit(gpu, odd, periodic, is_ij):
    n = 700
    box = np.array([1.0, 0.5, 0.125])
    r = np.random.default_rng(11)
    x = r.uniform(size=(n, 3)) * box
    x[: n // 3] = x[: n // 3] * 0.05 + 0.01             # a dense corner: windows of very different extents
    h = 0.05 * r.uniform(0.2, 1.0, n)
    if odd == "wide":
        h[::50] = 2.0
    if odd == "infinite":
        h[7] = np.inf
    if odd == "small":
        h[::3] *= 2.0 ** -60
    ref = _lists(gpu, x, h, box, periodic, 1.0, is_ij, 1)
    for log2_unit in (0, 60, 63, 100, 127, 130, 200, 300, -60, -75, -100, -150, -200, -300):
        got = _lists(gpu, x, h, box, periodic, 2.0 ** log2_unit, is_ij, 0)
        for i, (a, b) in enumerate(zip(got, ref)):
            np.testing.assert_array_equal(a, b, err_msg=f"2^{log2_unit}, particle {i}")
