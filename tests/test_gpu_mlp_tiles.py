"""Inference and training kernels at the edges of their row tiles (16 rows per
warp, 128 per training block, several rounds of the grid) against the FP64
oracle of the bf16 model: outputs, loss, gradient, and one Adam step.

Outputs agree to 2e-2 (the FP32 order of sums and SiLU's exponential move a bf16
rounding now and then).  Labels lie 1.5 or more above every output, so errors
y - t agree to 2e-2 / 1.5, the loss to twice that, and the gradients, whose dZ
the kernel rounds to bf16, to 3e-2 in the norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M():
    import mlp_oracle
    return mlp_oracle


@pytest.mark.parametrize("n", [1, 15, 17, 127, 129, 148 * 128 + 1])
def test_rows_at_tile_edges(gpu, M, n):
    states = M.random_states(n, seed=n)
    target = np.random.default_rng(n).uniform(2.0, 3.0, n)
    with gpu.Simulation(gpu.config_params("tube_gsph")) as sim:
        sim.mlp_init(3)
        params = sim.mlp_get_params()
        y = sim.mlp_predict(states)
        loss, grad = sim.mlp_train(states, np.exp(target) * states[:, 2], epochs=0)
    x = M.features(states)
    y_ref, _ = M.forward(params, x, emulate_bf16=True)
    assert np.max(y_ref) < 0.5
    assert np.max(np.abs(y - y_ref)) < 2e-2
    t = target.astype(np.float32).astype(np.float64)
    l_ref, g_ref = M.loss_and_grad(params, x, t, emulate_bf16=True)
    assert loss == pytest.approx(l_ref, rel=2.7e-2)
    for a, b in [(0, 320), (320, 384), (384, 4480), (4480, 4544), (4544, 8640), (8640, 8704), (8704, 8768),
                 (8768, 8769)]:
        assert np.linalg.norm(grad[a:b] - g_ref[a:b]) < 3e-2 * np.linalg.norm(g_ref[a:b])


def test_adam_steps_from_the_gradient(gpu, M):
    """One epoch of one batch: the first Adam step moves every parameter by lr
    g / (|g| + eps), and the network in use is the updated one."""
    n, lr = 1000, 1e-3
    states = M.random_states(n, seed=5)
    target = np.random.default_rng(5).uniform(2.0, 3.0, n)
    label = np.exp(target) * states[:, 2]
    with gpu.Simulation(gpu.config_params("tube_gsph")) as sim:
        sim.mlp_init(3)
        before = sim.mlp_get_params()
        _, grad = sim.mlp_train(states, label, epochs=0)
        sim.mlp_train(states, label, epochs=1, batch=n, lr=lr)
        after = sim.mlp_get_params()
        y = sim.mlp_predict(states)
    big = np.abs(grad) > 1e-3 * np.max(np.abs(grad))
    step = (after - before)[big]
    # m / c1 = g and sqrt(v / c2) = |g| in FP32: a few roundings of each, and the
    # subtraction's of a parameter below 1
    np.testing.assert_allclose(step, -lr * np.sign(grad[big]), atol=2e-4 * lr + 2.0 ** -24)
    y_ref, _ = M.forward(after, M.features(states), emulate_bf16=True)
    assert np.max(np.abs(y - y_ref)) < 2e-2


def test_workspace_kept_between_calls(gpu, M):
    """Calls of rising and falling size on one context, past the size whose
    workspace is kept (64 MB, 84 bytes a row): the outputs of a fresh context."""
    with gpu.Simulation(gpu.config_params("tube_gsph")) as sim:
        sim.mlp_init(3)
        for n in (100, 900_000, 40_000, 7):
            states = M.random_states(n, seed=n)
            y = sim.mlp_predict(states)
            loss, grad = sim.mlp_train(states, states[:, 2], epochs=0)
            with gpu.Simulation(gpu.config_params("tube_gsph")) as fresh:
                fresh.mlp_init(3)
                np.testing.assert_array_equal(y, fresh.mlp_predict(states))
                loss_f, grad_f = fresh.mlp_train(states, states[:, 2], epochs=0)
            # sums over blocks in any order: 148 FP32 additions
            assert loss == pytest.approx(loss_f, rel=148 * 2.0 ** -24)
            assert np.max(np.abs(grad - grad_f)) <= 148 * 2.0 ** -24 * np.max(np.abs(grad_f))
