"""Divisors whose significand is all ones, the exception of the corrected reciprocal
of csrc/rounded.cuh: the operations against CUDA's rounded ones (a program of its
own, built here), and the gravity walk's potential and acceleration bit for bit
against the oracle's at distances whose root, or whose 15-fold or cube, is one."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def counts(gpu, tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path_factory.mktemp("rounded") / "rounded_ops")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-I" + os.path.join(PKG, "csrc"), os.path.join(ROOT, "tests", "cpp", "rounded_ops.cu"), "-o", exe],
                   check=True)
    out = subprocess.run([exe, str(1 << 26)], check=True, capture_output=True, text=True, timeout=300).stdout
    return [(w[0], w[1], int(w[2]), *map(int, w[3:])) for w in (line.split() for line in out.splitlines())]


@pytest.mark.parametrize("kind", ["random", "near", "hard", "ones"])
def test_operations_round_as_cuda(counts, kind):
    rows = [r for r in counts if r[1] == kind]
    assert len(rows) >= 4
    for op, _, span, tested, refused, wrong, far in rows:
        assert far == 0 and tested > 1_000_000 and refused < tested // 2, (op, span, refused)
        if kind == "hard":
            # next to the middle of two doubles: the quotient from an unrounded
            # reciprocal and the root's reciprocal may miss, one in ten million
            assert wrong <= tested // 1_000_000, (op, span, wrong)
        elif kind != "ones" or op in ("any", "root", "rsqrt"):
            # (a quotient by a significand of all ones may be a unit off)
            assert wrong == 0, (op, span, wrong)


def _offsets(target, count, seed):
    """Offsets whose squared length, summed as the walk does, is `target`."""
    r = np.random.default_rng(seed)
    found = []
    while len(found) < count:
        x, z = r.uniform(0.1, 0.6, 4096), r.uniform(0.1, 0.5, 4096)
        y = np.sqrt(np.maximum(target - x * x - z * z, 0.0))
        for k in range(-4, 5):
            yk = y + k * np.spacing(y)
            ok = (x * x + yk * yk) + z * z == target
            found += list(zip(x[ok], yk[ok], z[ok]))
    return np.array(found[:count])


@pytest.mark.parametrize("theta", [0.1, 0.95])
@pytest.mark.parametrize("h", [0.05, 0.7, 3.0])
@pytest.mark.parametrize("what", ["root", "square", "fifteenfold", "cube"])
def test_gravity_at_odd_distances(gpu, O, what, h, theta):
    one = 1.0 - 2.0 ** -53
    if what == "root":
        targets = [one * one]
    elif what == "square":
        targets = [one]
    else:
        # roots r near a / 15, or near a cube root, whose product's low word is all ones
        r = np.random.default_rng(4)
        base = r.uniform(0.95, 1.0, 4_000_000)
        f = 15.0 * base if what == "fifteenfold" else base * base * base
        step = 15.0 if what == "fifteenfold" else 3.0 * base * base
        # move r so that the product's low 32 bits become ones
        bits = f.view(np.uint64) | np.uint64(0xffffffff)
        want = bits.view(np.float64)
        root = base + (want - f) / step
        got = 15.0 * root if what == "fifteenfold" else root * root * root
        root = root[(got.view(np.uint64) & np.uint64(0xffffffff)) == 0xffffffff]
        assert len(root) > 20
        targets = [x * x for x in root[:200] if np.sqrt(x * x) == x][:20]
    assert targets
    for t in targets:
        for d in _offsets(t, 1 if len(targets) > 1 else 8, 9):
            f = {"pos_x": np.array([0.0, d[0]]), "pos_y": np.array([0.0, d[1]]), "pos_z": np.array([0.0, d[2]]),
                 "mass": np.array([1.0, 1.5]), "sml": np.array([h, 1.2 * h])}
            p = gpu.config_params("evrard_ssph", theta=theta)
            o = O.Oracle(p, f)
            o.tree_make()
            o.gravity_force()
            ref = o.download(["acc_x", "acc_y", "acc_z", "phi"])
            with gpu.Simulation(p) as sim:
                sim.upload(f)
                sim.tree_make()
                sim.gravity_force()
                out = sim.download(list(ref))
            for k in ref:
                np.testing.assert_array_equal(out[k], ref[k], err_msg=f"{k} at {d}")
