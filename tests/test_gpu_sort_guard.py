"""The key sort's bounded wait: a tile whose predecessor never reports gives up,
sets its status bit and leaves the output in bounds (a program of its own, whose
one block is handed the second tile), and the bit comes back as an error of the
next call that waits, after which the context is usable."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu


def test_wait_for_a_tile_that_never_reports_ends(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "sort_wait")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-I" + os.path.join(PKG, "csrc"), "-I" + os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "sort_wait.cu"), "-o", exe], check=True)
    flag, ms, strange = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout.split()
    assert int(flag) == 16 and int(strange) == 0
    assert 1.0 < float(ms) < 20_000.0


def test_sort_guard_is_reported_at_the_next_wait(gpu):
    p = gpu.config_params("evrard_ssph")
    f = gpu.sample_evrard(8)
    with gpu.Simulation(p) as sim:
        sim.upload(f)
        sim.initialize()
        want = sim.download(["acc_x"])["acc_x"]
        assert gpu.lib().sphgpu_test_flag_pass_guard(sim._h, 16) == 0
        with pytest.raises(gpu.SPHException, match="key sort"):
            sim.synchronize()
        sim.synchronize()                      # reported once, then cleared
        assert gpu.lib().sphgpu_test_flag_pass_guard(sim._h, 16) == 0
        with pytest.raises(gpu.SPHException, match="key sort"):
            sim.tree_make()                    # its nodes are not built from unsorted keys
        with pytest.raises(gpu.SPHException, match="before tree"):
            sim.pre_interaction()
        sim.upload(f)
        sim.initialize()
        np.testing.assert_array_equal(sim.download(["acc_x"])["acc_x"], want)
