"""The temperature ladder on the GPU (k_thermo, csrc/thermo.cu) over the forms of its input: levels in
shared memory and in global memory, fewer levels than a warp, energies or temperatures that rule the
single-precision pass out, columns with and without counts -- against 64-bit NumPy.  Tolerance: an
exponent's own rounding, |E| / T and ln g to 2^-52 each, times the spread of what is averaged, plus 1e-13."""
import numpy as np
import pytest

CASES = [
    # levels, N, energy scale, Tmin, Tmax, temperatures, columns, counts column, trapezoid
    (2, 4, 8.0, 0.5, 5.0, 7, 0, -1, True), (31, 16, 32.0, 0.1, 10.0, 33, 3, 2, False),
    (33, 16, 32.0, 0.01, 50.01, 200, 1, -1, True), (1000, 1024, 2048.0, 0.01, 50.01, 1000, 17, 16, True),
    (4352, 4096, 8192.0, 0.05, 20.0, 300, 4, 3, True), (4353, 4096, 8192.0, 0.05, 20.0, 300, 4, 3, False),
    (20001, 4096, 8192.0, 0.5, 50.0, 100, 5, 4, True), (500, 256, 1e9, 0.01, 1.0, 50, 2, 1, True),
    (500, 256, 1e20, 1e17, 1e19, 50, 2, -1, True), (300, 1, 1e-9, 0.01, 1.0, 20, 1, -1, False),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=[f"{c[0]}x{c[5]}" for c in CASES])
def test_ladder(engine_lib, case):
    from rewl_simulator_gb300.thermo import thermodynamics
    nb, N, scale, Tmin, Tmax, nT, K, counts, trap = case
    rng = np.random.default_rng(nb)
    E = np.sort(rng.uniform(-scale, scale, nb))
    lng = 0.69 * N * (1 - (E / scale) ** 2) + rng.normal(0, 0.05, nb)
    obs = rng.uniform(0.1, 1.0, (nb, K)) if K else None
    if counts >= 0:
        obs[:, counts] = rng.integers(1, 10**6, nb)
    T, out = thermodynamics(E, lng, N, obs=obs, counts_col=counts, Tmin=Tmin, Tmax=Tmax, num_T=nT, trapezoid=trap)
    half = np.ones(nb)
    if trap:
        half[[0, -1]] = 0.5
    eps = 2.0 ** -52
    for i, t in enumerate(T):
        assert t == Tmin + (Tmax - Tmin) / nT * i
        x = lng - E / t
        m = x.max()
        w = np.exp(x - m) * half
        Z = w.sum()
        p = w / Z
        rel = 8 * eps * (np.abs(E).max() / t + np.abs(lng).max()) + 1e-13       # of a weight
        U, U2, S = p @ E / N, p @ (E * E) / N**2, p @ lng / N
        assert abs(out[i, 0] + t * (m + np.log(Z)) / N) <= rel * t / N + 1e-13 * abs(out[i, 0])
        assert abs(out[i, 1] - U) <= rel * (p @ np.abs(E)) / N
        assert abs(out[i, 2] - U2) <= rel * U2
        assert abs(out[i, 3] - S) <= rel * (p @ np.abs(lng)) / N
        assert abs(out[i, 4] - N * (U2 - U * U) / t**2) <= 4 * rel * N * U2 / t**2
        for k in range(K):
            ref = obs[:, k].mean() if k == counts else p @ obs[:, k]
            assert abs(out[i, 5 + k] - ref) <= rel * ref


@pytest.mark.gpu
def test_ground_state_at_zero_energy(engine_lib):
    """Energies from 0 to 10^9 at temperatures of order 1: the integers that span them are coarser than
    FP64 near the ground state, and the ladder keeps FP64's precision there."""
    from rewl_simulator_gb300.thermo import thermodynamics
    nb = 700
    E = np.concatenate([[0.0, 0.3, 0.7, 1.1, 1.9, 2.3], np.geomspace(3.0, 1e9, nb - 6)])
    lng = np.log1p(E)
    T, out = thermodynamics(E, lng, 16, Tmin=0.1, Tmax=4.1, num_T=40, trapezoid=False)
    for i, t in enumerate(T):
        x = lng - E / t
        w = np.exp(x - x.max())
        U = (w * E).sum() / w.sum() / 16
        assert abs(out[i, 1] - U) <= 4e-15 * U + 1e-300
