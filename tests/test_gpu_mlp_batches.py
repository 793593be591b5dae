"""The network's buffers over changing batch sizes: a gradient and a prediction do not depend on
what the network's buffers were grown for before, on the number of splits of the batch, or on
which rows the padding held."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, seed=5):
    rng = np.random.default_rng(seed)
    X = rng.normal(size=(n, 7)).astype(np.float32)
    return X, (X[:, 0] * X[:, 1] + 0.3).astype(np.float32)


def _fresh(layers, hidden, batch, X, y):
    from rewl_simulator_gb300.mlp import MLP
    m = MLP(hidden=hidden, layers=layers, seed=11)
    loss = m.gradient(X[:batch], y[:batch])
    out = loss, m.grads(), m.predict(X[:1])
    m.close()
    return out


# splits of the batch: 1024 and 4096 have some, 1152 and 4224 (larger) none
@pytest.mark.parametrize("hidden,layers,grown,batch", [(64, 1, 1152, 1024), (256, 4, 1061, 1024), (128, 2, 4224, 4096),
                                                       (128, 3, 4097, 128)])
def test_gradient_after_growth_equals_fresh(hidden, layers, grown, batch):
    from rewl_simulator_gb300.mlp import MLP
    X, y = _data(max(grown, batch))
    m = MLP(hidden=hidden, layers=layers, seed=11)
    m.gradient(X[:128], y[:128])
    m.predict(X[:grown])
    loss, g = m.gradient(X[:batch], y[:batch]), m.grads()
    p = m.predict(X[:1])
    m.close()
    floss, fg, fp = _fresh(layers, hidden, batch, X, y)
    assert loss == floss and np.array_equal(g, fg) and np.array_equal(p, fp)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000])
def test_prediction_rows_do_not_depend_on_padding(n):
    from rewl_simulator_gb300.mlp import MLP
    X, _ = _data(1500)
    m = MLP(hidden=64, layers=2, seed=3)
    whole = m.predict(X)
    assert np.array_equal(m.predict(X[:n]), whole[:n])
    m.close()
