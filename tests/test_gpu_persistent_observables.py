"""The persistent launch with observables: an uneven batch (Ising on the bin-tracking and on the global-table form,
Ashkin-Teller on the tree) follows the trajectories of the launch groups on their streams, with the same averages."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("graphs", [0, 1])
@pytest.mark.parametrize("obs", [1, 2])
def test_uneven_batch(engine_lib, obs, graphs):
    rg = engine_lib
    h = np.round(np.random.default_rng(2).normal(0, 0.5, 49) * 2**20) / 2**20

    def engine(persistent):
        ising = dict(model=rg.MODEL_ISING2D, num_windows=3, replicas_per_window=3, init_mode=0)
        inss = [rg.Instance(L=12, energy_min=-288.0, energy_max=292.0, bin_width=4.0, seed=1, **ising),
                rg.Instance(L=20, energy_min=-800.0, energy_max=804.0, bin_width=4.0, seed=2, **ising),
                rg.Instance(L=10, energy_min=-200.0, energy_max=208.0, bin_width=8.0, seed=3, **ising),
                rg.Instance(model=rg.MODEL_ASHKIN_TELLER2D, L=7, K=0.5, fields=h, energy_min=-245.0, energy_max=0.0, bin_width=0.05,
                            num_windows=2, replicas_per_window=4, seed=4)]
        return rg.Engine(rg.Batch(instances=inss, sweeps_per_exchange=25, sweeps_per_check=50, mask_mode=rg.MASK_VISITED, observables=obs,
                                  graphs=graphs, persistent=persistent))
    with engine(1) as a, engine(0) as b:
        for e in (a, b):
            e.run_cycles(3)
        for w in range(b.num_walkers):
            x, y = a.export_walker(w), b.export_walker(w)
            for k in x:
                assert np.array_equal(x[k], y[k]), (w, k)
        for i, windows in enumerate(b.windows):
            for w in range(len(windows)):
                x, y = a.window_observables(i, w), b.window_observables(i, w)
                assert np.array_equal(x[:, -1], y[:, -1])
                # sums of at most 4 x 150 x 400 terms in another order, to 2^-53 of the sum each; transforms to 60 places
                np.testing.assert_allclose(x, y, rtol=4 * 150 * 400 * 2.0**-53, atol=1e-13)
