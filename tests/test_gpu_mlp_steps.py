"""The training cursor on the device: steps of one call are those of as many calls of one step each, bit for bit
(the kernel that sums a step's loss moves the cursor on, between the kernels that read it, csrc/mlp.cu)."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("hidden, layers, steps", [(64, 1, 40), (256, 4, 24), (512, 5, 12)])
def test_steps_of_one_call_equal_single_steps(engine_lib, hidden, layers, steps):
    from rewl_simulator_gb300.mlp import MLP
    r = np.random.default_rng(5)
    X, y = r.uniform(-1, 1, (700, 7)).astype(np.float32), r.uniform(0, 1, 700).astype(np.float32)
    a, b = (MLP(hidden=hidden, layers=layers, seed=3) for _ in range(2))
    for m in (a, b):
        m.set_data(X, y)
    together = a.train(steps, batch=128, lr=1e-3)
    single = np.concatenate([b.train(1, batch=128, lr=1e-3) for _ in range(steps)])
    assert np.array_equal(together, single)
    assert np.array_equal(a.params(), b.params())
    assert len(set(together.tolist())) > steps // 2            # (each step keeps its own loss)
