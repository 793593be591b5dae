"""Launch shapes of the bin-tracking Ising kernel by what an SM holds (shape_bins, csrc/engine.cu): walkers per warp, with
and without visits beside g, moments in shared or global memory, the form of fewer registers in crowded launches.  A
walker's trajectory does not depend on its launch: the first instance of a large batch equals an engine of its own."""
import numpy as np
import pytest

CASES = [
    # L, windows, replicas, instances, observables, walkers per warp expected
    (64, 16, 64, 2, 0, 4), (64, 16, 64, 2, 1, 2), (64, 16, 64, 2, 2, 2), (64, 4, 64, 4, 0, 1), (64, 1, 64, 10, 0, 1), (64, 8, 64, 4, 0, 4),
    (16, 8, 8, 46, 1, 2), (16, 8, 8, 46, 2, 2), (16, 8, 8, 93, 0, 4), (16, 8, 8, 93, 1, 4), (16, 8, 8, 93, 2, 4), (20, 6, 8, 14, 1, 1),
]


def _engine(rg, L, windows, replicas, instances, obs, **kw):
    inss = [rg.Instance(model=rg.MODEL_ISING2D, L=L, energy_min=-2.0 * L * L, energy_max=2.0 * L * L + 4, bin_width=4.0, num_windows=windows,
                        replicas_per_window=replicas, init_mode=0, seed=900 + 7 * i) for i in range(instances)]
    return rg.Engine(rg.Batch(instances=inss, sweeps_per_exchange=4, sweeps_per_check=8, observables=obs, **kw))


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=lambda c: "L%d_%dx%dx%d_obs%d" % c[:5])
def test_first_instance_of_a_large_batch(engine_lib, case):
    rg = engine_lib
    L, windows, replicas, instances, obs, per_warp = case
    with _engine(rg, L, windows, replicas, instances, obs) as a, \
            _engine(rg, L, windows, replicas, 1, obs, walkers_per_warp=1) as b:
        assert tuple(a.launch_shapes()[0][1:3]) == (1, per_warp)
        assert tuple(b.launch_shapes()[0][1:3]) == (1, 1)
        for e in (a, b):
            e.run_cycles(2)
        for w in range(0, b.num_walkers, max(1, b.num_walkers // 17)):
            x, y = a.export_walker(w), b.export_walker(w)
            for k in x:
                assert np.array_equal(x[k], y[k]), (w, k)
        for w in range(windows if obs else 0):
            x, y = a.window_observables(0, w), b.window_observables(0, w)
            assert np.array_equal(x[:, -1], y[:, -1])
            # sums of at most 64 x 16 L^2 terms in another order, to 2^-53 of the sum each
            np.testing.assert_allclose(x, y, rtol=64 * 16 * L * L * 2.0**-53, atol=1e-300)


@pytest.mark.gpu
@pytest.mark.parametrize("obs", [0, 1, 2])
@pytest.mark.parametrize("per_warp", [1, 2, 4])
def test_walkers_per_warp_is_kept_where_it_fits(engine_lib, per_warp, obs):
    """One window of 4,097 bins: four walkers fit a block's 200 KB without visits beside g (8 bytes a bin), with the
    correlators' counts (12 bytes a bin) two."""
    rg = engine_lib
    with _engine(rg, 64, 1, 4, 1, obs, walkers_per_warp=per_warp) as a, _engine(rg, 64, 1, 4, 1, obs, walkers_per_warp=1) as b:
        assert a.launch_shapes()[0][2] == (min(per_warp, 2) if obs == 2 else per_warp)
        for e in (a, b):
            e.run_cycles(2)
        for w in range(4):
            x, y = a.export_walker(w), b.export_walker(w)
            for k in x:
                assert np.array_equal(x[k], y[k]), (w, k)


@pytest.mark.gpu
@pytest.mark.parametrize("obs", [0, 1, 2])
@pytest.mark.parametrize("per_warp", [0, 2, 4])
@pytest.mark.parametrize("L, windows, J", [(4, 1, 1.0), (8, 4, 1.0), (8, 3, -1.0), (16, 8, 1.0)])
def test_short_rows_one_decision_after_another(engine_lib, L, windows, J, per_warp, obs):
    """Rows of 4, 8 and 16 sites in launches of more walkers than schedulers (k_sweep_ising_rows): the first instance of
    such a batch equals an engine of its own, whose walkers go through the tree.  (J = -1 turns the energies around;
    enough visits for several transforms of the correlators.)"""
    rg = engine_lib
    N = L * L

    def engine(instances, **kw):
        inss = [rg.Instance(model=rg.MODEL_ISING2D, L=L, J=J, energy_min=-2.0 * N, energy_max=2.0 * N + 4, bin_width=4.0, num_windows=windows,
                            replicas_per_window=8, init_mode=0, seed=40 + i) for i in range(instances)]
        return rg.Engine(rg.Batch(instances=inss, sweeps_per_exchange=33, sweeps_per_check=99, observables=obs, **kw))
    with engine(640 // (8 * windows) + 1, walkers_per_warp=per_warp) as a, engine(1, walkers_per_warp=1) as b:
        # (L = 16 with correlators stays with the tree, whose choice is one walker a warp here)
        assert a.launch_shapes()[0][2] in ((per_warp,) if per_warp else (1,) if L == 16 and obs == 2 else (2, 4))
        for _ in range(3):
            for e in (a, b):
                e.run_cycles(1)
            for w in range(b.num_walkers):
                x, y = a.export_walker(w), b.export_walker(w)
                for k in x:
                    assert np.array_equal(x[k], y[k]), (w, k)
        for w in range(windows if obs else 0):
            x, y = a.window_observables(0, w), b.window_observables(0, w)
            assert np.array_equal(x[:, -1], y[:, -1])
            # sums of at most 8 x 297 N terms in another order, to 2^-53 of the sum each; the table of the
            # correlators' transforms holds 60 places
            np.testing.assert_allclose(x, y, rtol=8 * 297 * N * 2.0**-53, atol=1e-13)
