"""Positions of the global-table kernel's decision tree in 32 bits: bin widths with and without common
binary zeros, and single flips just within and just beyond what they hold, against the oracle."""
import numpy as np
import pytest

from test_gpu_parity import _compare, _pair

# L, bin width, field of one site, energies
CASES = [
    (6, 0.05, 44.0, -224.0, -20.0), (6, 0.05, 48.0, -228.0, -20.0),      # 100 energy units: the limit lies between
    (5, 1.0, 240.0, -365.0, -200.0), (5, 1.0, 260.0, -385.0, -200.0),    # 500
    (7, 1.0 / 3.0, 0.5, -246.0, 0.0), (8, 1.0 / 64.0, 0.5, -330.0, -100.0), (6, 1.0 / 4095.0, 0.0, -180.0, -90.0),
    (9, 1.0 / 4096.0, 0.25, -410.0, -300.0), (33, 0.2, 0.5, -5500.0, -200.0),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"L{c[0]}_bw{c[1]:.4g}_h{c[2]:g}")
def test_positions_match_the_oracle(engine_lib, oracle_lib, case):
    L, bw, field, lo, hi = case
    h = np.zeros(L * L)
    if field:
        h[::5] = 0.25
        h[7] = field
    eng, orc = _pair(engine_lib, oracle_lib, 1, L, lo, hi, bw, 2, 2, 6, 12, 900 + L, K=0.5, fields=h if field else None, mask=1)
    try:
        for k in range(2):
            eng.run_cycles(1)
            orc.cycle()
            _compare(eng, orc, f"cycle {k}")
    finally:
        eng.close()
        orc.close()


@pytest.mark.gpu
@pytest.mark.parametrize("more", [0, 1])
def test_crowded_launches_with_observables_run_the_same_trajectories(engine_lib, more):
    """With observables, more than seven walkers per SM decide serially: an instance's tables and
    averages are those of an engine of its own, on either side of the line."""
    import torch
    rg = engine_lib
    n = 7 * torch.cuda.get_device_properties(0).multi_processor_count + more
    counts = [4] + [64] * ((n - 4) // 64) + ([(n - 4) % 64] if (n - 4) % 64 else [])
    h = np.round(np.random.default_rng(3).normal(0, 0.5, 25) * 2**20) / 2**20

    def engine(cs):
        inss = [rg.Instance(model=rg.MODEL_ASHKIN_TELLER2D, L=5, K=0.5, fields=h, energy_min=-125.0, energy_max=0.0, bin_width=0.05,
                            num_windows=1, replicas_per_window=r, seed=70 + i) for i, r in enumerate(cs)]
        return rg.Engine(rg.Batch(instances=inss, sweeps_per_exchange=20, sweeps_per_check=40, mask_mode=rg.MASK_VISITED,
                                  observables=2))
    with engine(counts) as a, engine(counts[:1]) as b:
        for e in (a, b):
            e.run_cycles(2)
        assert np.array_equal(a.window_logdos(0, 0), b.window_logdos(0, 0))
        x, y = a.window_observables(0, 0), b.window_observables(0, 0)
        assert np.array_equal(x[:, -1], y[:, -1])
        # sums of at most 4000 terms in another order: 4000 x 2^-53 of the larger
        np.testing.assert_allclose(x, y, rtol=1e-11, atol=1e-13)
