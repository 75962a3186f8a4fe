"""The pair lists' finalise pass at the sizes where the rows of one warp change
(1, 2, 4 .. of them): a centrally graded cloud, whose inner rows get tails of
more than 32 entries, against the pairs r < max(h_i, h_j) of a k-d tree."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FILL = 148 * 32


@pytest.mark.parametrize("n", [2, 33, 2 * FILL - 1, 2 * FILL, 4 * FILL + 5])
def test_rows_per_warp(gpu, n):
    spatial = pytest.importorskip("scipy.spatial")
    r = np.random.default_rng(n)
    u = r.standard_normal((n, 3))
    x = u / np.linalg.norm(u, axis=1)[:, None] * r.uniform(0.0, 1.0, n)[:, None] ** 2
    f = {f"pos_{a}": x[:, k].copy() for k, a in enumerate("xyz")}
    rad = np.maximum(np.linalg.norm(x, axis=1), 0.05)
    f["mass"] = np.full(n, 1.0 / n)
    f["dens"] = 1.0 / (8.0 * np.pi * rad ** 2.5)
    f["ene"] = np.ones(n)
    f["sound"] = np.ones(n)
    f["alpha"] = np.ones(n)
    with gpu.Simulation(gpu.config_params("evrard_ssph", use_gravity=0, iterative_sml=0)) as sim:
        sim.upload(f)
        sim.initialize()
        sim.tree_make()
        sim.pre_interaction()
        off, ids = sim.force_pairs()
        st = sim.download(["pos_x", "pos_y", "pos_z", "sml"])
    x = np.stack([st[f"pos_{a}"] for a in "xyz"], 1)
    h = st["sml"]
    near = spatial.cKDTree(x).query_ball_point(x, h * (1.0 + 1e-9))
    want = [set() for _ in range(n)]
    longest = 0
    for i in range(n):
        j = np.array(near[i])
        d = x[i][None, :] - x[j]
        j = j[np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]) < h[i]]
        want[i].update(j.tolist())
        for k in j.tolist():
            want[k].add(i)
    for i in range(n):
        got = ids[off[i]:off[i + 1]].tolist()
        assert len(got) == len(set(got)) and set(got) == want[i], i
        d = x[i][None, :] - x[got]
        longest = max(longest, int(np.sum(np.sqrt((d * d).sum(1)) > h[i] * (1.0 + 1e-9))))
    assert n < 1000 or longest > 32
