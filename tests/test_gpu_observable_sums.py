"""Per-bin moments kept as whole numbers across many visits, and correlators by groups of lanes,
against the oracle's sums (the tolerance of the observables' parity tests)."""
import numpy as np
import pytest

from test_gpu_parity import _run_observables_case

# name, model, L, energies, bin width, windows, replicas, sweeps per exchange / check, seed, cycles, walkers per warp,
# field width, mask, observables
CASES = [
    # more visits in a launch than the moments' words hold (2^14): booked on the way
    ("ising_L8_booked_1", 0, 8, -128.0, 132.0, 4.0, 1, 2, 700, 700, 41, 1, 1, 0.0, 0, 1),
    ("ising_L8_booked_2", 0, 8, -128.0, 132.0, 4.0, 1, 3, 700, 700, 42, 1, 2, 0.0, 0, 2),
    ("ising_L10_booked_4", 0, 10, -200.0, 204.0, 4.0, 2, 3, 400, 400, 43, 1, 4, 0.0, 0, 2),
    # transforms in the first visits of many bins, planes longer and shorter than a group of lanes
    ("ising_L3", 0, 3, -18.0, 2.0, 4.0, 1, 3, 600, 600, 44, 2, 4, 0.0, 0, 2),
    ("ising_L33", 0, 33, -2178.0, 2.0, 4.0, 3, 2, 4, 8, 45, 2, 2, 0.0, 0, 2),
    ("at_L5", 1, 5, -125.0, 0.0, 0.05, 1, 2, 100, 200, 46, 2, 0, 0.5, 1, 2),
    ("at_L8", 1, 8, -320.0, 0.0, 0.05, 2, 2, 40, 80, 47, 2, 0, 0.5, 1, 2),
    ("at_L16", 1, 16, -1280.0, 0.0, 0.05, 2, 2, 10, 20, 48, 2, 0, 0.5, 1, 2),
    ("at_L34", 1, 34, -5780.0, 0.0, 0.5, 2, 1, 3, 6, 49, 1, 0, 0.5, 1, 2),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_observable_sums_match_the_oracle(engine_lib, oracle_lib, case):
    _run_observables_case(engine_lib, oracle_lib, case)


def test_table_entries_in_two_parts_are_closer_than_their_rounding():
    """cos and sin as hi 2^-30 + lo 2^-60 (both 32-bit) differ from the FP64 entries by less than the
    entries' own rounding error where they are 1/2 or more, and by 2^-61 at most elsewhere."""
    for L in range(2, 129):
        x = np.arange(L) * (2.0 * np.arccos(-1.0) / L)
        c = np.concatenate([np.cos(x), np.sin(x)])
        units = np.ldexp(c, 30)
        hi = np.rint(units)
        lo = np.rint(np.ldexp(units - hi, 30))
        assert np.all(np.abs(hi) <= 2**30) and np.all(np.abs(lo) <= 2**29)
        err = np.ldexp(units - hi, 30) - lo                    # in units of 2^-60, exact
        assert np.all(np.abs(err) <= 0.5)


def test_root_of_whole_numbers_by_two_newton_steps():
    """x^2 = k from a reciprocal root good to 2 units of single precision either way, restated with exact
    residuals: the FP64 root to one unit in the last place."""
    from fractions import Fraction
    rng = np.random.default_rng(1)
    ks = [1, 2, 3, 4, 5, 2**20 + 1, 2**28 - 1, 2 * 16384**2] + [int(k) for k in rng.integers(1, 2 * 16384**2, 1500)]
    for k in ks:
        for off in (-2, 0, 2):
            y = np.float32(1.0 / np.sqrt(float(k)))
            y = np.float32(y + off * np.spacing(y))
            half, x = float(np.float32(0.5) * y), float(np.float32(k) * y)
            for _ in range(2):
                r = float(Fraction(k) - Fraction(x) * Fraction(x))
                x = float(Fraction(x) + Fraction(r) * Fraction(half))
            assert abs(x - np.sqrt(float(k))) <= np.spacing(np.sqrt(float(k)))
