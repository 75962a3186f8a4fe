"""Device memory of a context: what only the FP64 gravity walk reads (32 bytes a
particle) is not held by a mixed run that never re-evaluates in FP64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _held(gpu, f, **kw):
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with gpu.Simulation(gpu.config_params("evrard_ssph", **kw)) as sim:
        sim.upload(f)
        sim.synchronize()
        return before - torch.cuda.mem_get_info()[0]


def test_mixed_gravity_holds_no_fp64_half_kernels(gpu):
    n = 1_000_000
    r = np.random.default_rng(1)
    f = {f"pos_{a}": r.uniform(size=n) for a in "xyz"}
    f["mass"] = np.full(n, 1.0 / n)
    _held(gpu, f, precision=gpu.MIXED)     # the first context pays for what the library itself loads
    plain = _held(gpu, f, precision=gpu.MIXED, use_gravity=0)
    mixed = _held(gpu, f, precision=gpu.MIXED)
    again = _held(gpu, f, precision=gpu.MIXED, mixed_acc_tol=1e-3)
    assert mixed - plain < 16 * n
    assert again - plain >= 32 * n        # re-evaluating, it needs them
