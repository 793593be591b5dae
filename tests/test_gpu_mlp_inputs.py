"""Inputs larger than the network's staging buffer (upload_features, csrc/mlp.cu): predictions as in pieces, and a training
set held once."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("in_dim, n", [(64, 65536), (64, 65537), (64, 150000), (7, 600001)])
def test_predictions_in_pieces(engine_lib, in_dim, n):
    from rewl_simulator_gb300.mlp import MLP
    m = MLP(hidden=64, layers=1, seed=3)
    X = np.random.default_rng(n).uniform(-1, 1, (n, in_dim)).astype(np.float32)
    y = m.predict(X)
    for i in range(0, n, 40000):
        assert np.array_equal(y[i:i + 40000], m.predict(X[i:i + 40000]))


@pytest.mark.gpu
def test_training_set_is_held_once(engine_lib):
    import torch
    from rewl_simulator_gb300.mlp import MLP
    n = 2_000_000
    m = MLP(hidden=64, layers=1, seed=3)
    X, y = np.zeros((n, 64), dtype=np.float32), np.zeros(n, dtype=np.float32)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    m.set_data(X, y)
    # 64 bf16 inputs and a target a row, the staging buffer, and the allocator's granularity
    assert before - torch.cuda.mem_get_info()[0] <= n * (128 + 4) + (16 << 20) + (32 << 20)
