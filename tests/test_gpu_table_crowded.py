"""Crowded Ashkin-Teller launches on either side of the line between the tree and the serial chain (table_cache,
csrc/engine.cu): coarse bins, whose tables many walkers of an SM hold, and fine ones, of which few do.  An instance's
tables and averages are those of an engine of its own."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("obs", [0, 1, 2])
@pytest.mark.parametrize("bin_width, low, high", [(1.0, -180.0, 0.0), (0.05, -180.0, 0.0), (0.01, -150.0, -110.0)])
def test_first_instance_of_a_crowded_batch(engine_lib, bin_width, low, high, obs):
    rg = engine_lib
    h = np.round(np.random.default_rng(5).normal(0, 0.5, 36) * 2**20) / 2**20

    def engine(instances):
        inss = [rg.Instance(model=rg.MODEL_ASHKIN_TELLER2D, L=6, K=0.5, fields=h, energy_min=low, energy_max=high, bin_width=bin_width,
                            num_windows=1, replicas_per_window=20, seed=11 + i) for i in range(instances)]
        return rg.Engine(rg.Batch(instances=inss, sweeps_per_exchange=20, sweeps_per_check=40, mask_mode=rg.MASK_VISITED, observables=obs))
    with engine(64) as a, engine(1) as b:
        for e in (a, b):
            e.run_cycles(2)
        for w in range(0, 20, 3):
            x, y = a.export_walker(w), b.export_walker(w)
            for k in x:
                assert np.array_equal(x[k], y[k]), (w, k)
        if obs:
            x, y = a.window_observables(0, 0), b.window_observables(0, 0)
            assert np.array_equal(x[:, -1], y[:, -1])
            # sums of at most 20 x 80 x 72 terms in another order, to 2^-53 of the sum each; transforms to 60 places
            np.testing.assert_allclose(x, y, rtol=20 * 80 * 72 * 2.0**-53, atol=1e-13)
