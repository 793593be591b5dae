"""The bin-tracking kernel's decision tree on the GPU at the sizes where it can go wrong: rows of
one block, of two, with a short last block, rows cut into unequal chunks, one site per row short of
or beyond a word, two bins per neighbour, windows too large for visit counts in shared memory, and
the integer moment sums -- bit for bit against the oracle (moments to FP64 rounding)."""
import numpy as np
import pytest

from test_gpu_parity import _compare, _pair, _run_observables_case

# L, bin width, windows, replicas, sweeps per exchange / check, cycles
SIZES = [
    (3, 4.0, 1, 2, 50, 100, 3), (4, 4.0, 2, 2, 50, 100, 3), (5, 4.0, 2, 3, 40, 80, 3), (6, 2.0, 2, 5, 20, 40, 3),
    (9, 4.0, 3, 2, 20, 40, 3), (10, 4.0, 3, 3, 20, 40, 3), (11, 4.0, 2, 2, 10, 20, 3), (15, 2.0, 3, 2, 10, 20, 2),
    (20, 4.0, 4, 5, 10, 20, 2), (31, 4.0, 3, 2, 4, 8, 2), (33, 4.0, 3, 3, 4, 8, 2), (37, 4.0, 2, 2, 3, 6, 2),
    (66, 4.0, 2, 2, 2, 4, 2), (70, 4.0, 3, 2, 2, 4, 1), (127, 4.0, 2, 1, 1, 2, 1),
]


@pytest.mark.gpu
@pytest.mark.parametrize("walkers_per_warp", [1, 2, 4])
@pytest.mark.parametrize("case", SIZES, ids=lambda c: f"L{c[0]}_bw{c[1]:g}")
def test_lattice_sizes_match_the_oracle(engine_lib, oracle_lib, case, walkers_per_warp):
    L, bw, nwin, R, se, sc, cycles = case
    N = L * L
    top = 2.0 * N + 4 if L % 2 == 0 else 0.0 if (2 * N) % 4 == 0 else 2.0     # odd tori: the lower half
    top += -(top + 2 * N) % bw
    eng, orc = _pair(engine_lib, oracle_lib, 0, L, -2.0 * N, top, bw, nwin, R, se, sc, 100 + L,
                     walkers_per_warp=walkers_per_warp)
    try:
        assert eng.launch_shapes()[0][1] == 1                  # the bin-tracking kernel
        for k in range(cycles):
            eng.run_cycles(1)
            orc.cycle()
            _compare(eng, orc, f"cycle {k}")
    finally:
        eng.close()
        orc.close()


@pytest.mark.gpu
def test_window_without_room_for_visit_counts(engine_lib, oracle_lib):
    """12,802 bins: 16 bytes a bin do not fit a block's shared memory, 8 do."""
    eng, orc = _pair(engine_lib, oracle_lib, 0, 80, -12800.0, 12804.0, 2.0, 1, 3, 3, 6, 77, walkers_per_warp=2)
    try:
        shapes = eng.launch_shapes()
        assert shapes[0][1] == 1 and shapes[0][2] == 1         # g alone: one walker per warp
        for k in range(2):
            eng.run_cycles(1)
            orc.cycle()
            _compare(eng, orc, f"cycle {k}")
    finally:
        eng.close()
        orc.close()


OBS = [
    ("L5", 0, 5, -50.0, -6.0, 4.0, 2, 2, 40, 80, 31, 3, 0, 0.0, 0, 2),
    ("L20_2perwarp", 0, 20, -800.0, 804.0, 4.0, 4, 3, 20, 40, 33, 2, 2, 0.0, 0, 2),
    ("L33_4perwarp", 0, 33, -2178.0, -300.0 + 22, 4.0, 3, 3, 4, 8, 35, 2, 4, 0.0, 0, 2),
    # 12,802 bins: moments added in global memory
    ("L80_one_window", 0, 80, -12800.0, 12804.0, 2.0, 1, 2, 2, 4, 37, 2, 0, 0.0, 0, 1),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", OBS, ids=[c[0] for c in OBS])
def test_observables_match_the_oracle(engine_lib, oracle_lib, case):
    _run_observables_case(engine_lib, oracle_lib, case)


AT = [
    # L, K, sigma_h, bin width, windows, replicas, sweeps per exchange / check, observables
    (2, 0.5, 0.5, 0.05, 1, 2, 50, 100, 0), (3, 0.25, 0.3, 0.05, 2, 2, 40, 80, 0), (9, 0.75, 0.0, 0.25, 2, 2, 10, 20, 0),
    (10, 0.5, 0.5, 0.05, 3, 2, 10, 20, 2), (11, 0.5, 0.5, 1.0, 2, 2, 10, 20, 1), (17, 0.25, 0.3, 0.05, 4, 2, 4, 8, 0),
    (33, 0.5, 0.5, 0.05, 4, 2, 2, 4, 0), (37, 0.5, 0.5, 0.05, 3, 1, 2, 4, 1), (20, 0.5, 3.0, 0.0625, 2, 2, 4, 8, 0),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", AT, ids=lambda c: f"L{c[0]}_bw{c[3]:g}_obs{c[8]}")
def test_ashkin_teller_tree_matches_the_oracle(engine_lib, oracle_lib, case):
    """Whole-row and cut rows, one block and several, windows smaller and larger than the bins held
    in shared memory, strong fields (energy changes far beyond them)."""
    L, K, sig, bw, nwin, R, se, sc, obs = case
    _run_observables_case(engine_lib, oracle_lib, ("", 1, L, -5.0 * L * L, 0.0, bw, nwin, R, se, sc, 300 + L, 2, 0, sig, 1, obs)) \
        if obs else _at_case(engine_lib, oracle_lib, case)


def _at_case(rg, po, case):
    L, K, sig, bw, nwin, R, se, sc, _ = case
    h = np.round(np.random.default_rng(L).normal(0, sig, L * L) * 2**20) / 2**20 if sig else None
    eng, orc = _pair(rg, po, 1, L, -np.ceil(2 * (2 + K)) * L * L, 0.0, bw, nwin, R, se, sc, 300 + L, K=K, fields=h, mask=1)
    try:
        for k in range(2):
            eng.run_cycles(1)
            orc.cycle()
            _compare(eng, orc, f"cycle {k}")
    finally:
        eng.close()
        orc.close()


@pytest.mark.gpu
def test_fields_beyond_the_tree_run_the_serial_chain(engine_lib, oracle_lib):
    """One site's field carries an energy change across more than 2^26 bins: the launch group decides
    serially, and so it does when such fields are imported later."""
    rg, po = engine_lib, oracle_lib
    h = np.zeros(36)
    h[7] = 4.0e6
    big = dict(K=0.5, fields=h, mask=1)
    eng, orc = _pair(rg, po, 1, 6, -180.0 - 4.0e6, -4.0e6, 0.05, 2, 2, 10, 20, 61, **big)
    try:
        eng.run_cycles(1)
        orc.cycle()
        _compare(eng, orc, "created")
    finally:
        eng.close()
        orc.close()
    ins = rg.Instance(model=rg.MODEL_ASHKIN_TELLER2D, L=6, K=0.5, fields=np.zeros(36), energy_min=-180.0, energy_max=0.0,
                      bin_width=0.05, num_windows=2, replicas_per_window=2, seed=61)
    with rg.Engine(rg.Batch(instances=[ins], sweeps_per_exchange=10, sweeps_per_check=20, mask_mode=rg.MASK_VISITED)) as a, \
            rg.Engine(rg.Batch(instances=[ins], sweeps_per_exchange=10, sweeps_per_check=20, mask_mode=rg.MASK_VISITED)) as b:
        a.run_cycles(1)
        b.run_cycles(1)
        a.import_disorder(0, np.zeros(36))          # the same fields: still the tree
        h[7] = 4.0e6
        b.import_disorder(0, h)                     # serial from here on ...
        b.import_disorder(0, np.zeros(36))          # ... with the same energies as before
        for k in range(2):
            a.run_cycles(1)
            b.run_cycles(1)
        for s in range(4):
            x, y = a.export_walker(s), b.export_walker(s)
            for key in x:
                np.testing.assert_array_equal(x[key], y[key], err_msg=f"walker {s} {key}")
