"""The temperature ladder (rewl_thermodynamics, csrc/thermo.cu) on inputs at the edge of what it takes."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("level", [0, 150, 299])
@pytest.mark.parametrize("levels", [300, 5000])
def test_averages_that_are_not_finite(engine_lib, value, level, levels):
    """A column with a NaN or an infinity at one level averages to what its sum of products gives, whatever weight
    the level has: NaN, or an infinity where the level's weight is not zero.  The other columns are as without it."""
    from rewl_simulator_gb300.thermo import thermodynamics
    E = np.linspace(-2048.0, 2048.0, levels)
    lng = 700.0 * (1 - (E / 2048.0) ** 2)
    obs = np.random.default_rng(1).uniform(0.1, 1.0, (levels, 3))
    T, plain = thermodynamics(E, lng, 1024, obs=obs, counts_col=2, Tmin=0.05, Tmax=50.0, num_T=60)
    obs[level, 1] = value
    _, out = thermodynamics(E, lng, 1024, obs=obs, counts_col=2, Tmin=0.05, Tmax=50.0, num_T=60)
    keep = [0, 1, 2, 3, 4, 5, 7]
    np.testing.assert_allclose(out[:, keep], plain[:, keep], rtol=1e-9)
    zero = 0
    for i, t in enumerate(T):
        x = lng - E / t
        gap = x.max() - x[level]
        if abs(gap - 745.2) < 1.0:                 # between zero and the smallest subnormal, as the rounding goes
            continue
        zero += gap > 745.2
        with np.errstate(invalid="ignore"):
            ref = value * (0.0 if gap > 745.2 else 1.0)
        assert np.array_equal(out[i, 6], ref, equal_nan=True), (t, out[i, 6], ref)
    assert (zero > 0) == (level > 0)               # the ground state always counts, the others not at every temperature


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [0.0, 1e-300, 1e-30, 1e-18, 1e-15, 1e-12, 1e-9])
def test_flat_density_of_states(engine_lib, scale):
    """ln g of nearly nothing: the integer exponents keep every place that counts beside -E / T."""
    from rewl_simulator_gb300.thermo import thermodynamics
    r = np.random.default_rng(4)
    E = np.sort(r.uniform(-64.0, 64.0, 400))
    lng = scale * r.uniform(-1.0, 1.0, 400)
    T, out = thermodynamics(E, lng, 64, Tmin=0.5, Tmax=40.0, num_T=50, trapezoid=False)
    for i, t in enumerate(T):
        x = lng - E / t
        w = np.exp(x - x.max())
        rel = 8 * 2.0**-52 * 64 / t + 1e-13
        U = (w * E).sum() / w.sum() / 64
        assert abs(out[i, 0] + t * (x.max() + np.log(w.sum())) / 64) <= rel * t / 64 + 1e-13 * abs(out[i, 0])
        assert abs(out[i, 1] - U) <= rel * 64 / 64


@pytest.mark.gpu
@pytest.mark.parametrize("levels", [2, 33, 500, 4352, 4353])
@pytest.mark.parametrize("columns", [0, 5, 17])
def test_rows_do_not_depend_on_the_ladder(engine_lib, levels, columns):
    """A temperature's row is the same in a ladder that fills the device (a warp a temperature) and in short ones
    (teams of 2 to 16 warps a temperature), to the order of its sums: n terms, n x 2^-53 of the sum of magnitudes;
    for the specific heat N (U2 - U^2) / T^2 those of its two terms."""
    from rewl_simulator_gb300.thermo import thermodynamics
    r = np.random.default_rng(levels)
    E = np.linspace(-2.0, 2.0, levels) * 1024
    lng = 710.0 * (1 - (E / 2048.0) ** 2)
    obs = r.uniform(0.1, 1.0, (levels, columns)) if columns else None
    step, low = 1.0 / 128, 0.5

    def ladder(n):
        return thermodynamics(E, lng, 1024, obs=obs, counts_col=columns - 1, Tmin=low, Tmax=low + step * n, num_T=n)
    T, full = ladder(5000)
    size = np.abs(full).max(axis=0)
    for n in (1, 2, 151, 153, 305, 607, 609, 1217, 2433):
        t, rows = ladder(n)
        assert np.array_equal(t, T[:n])
        off = np.abs(rows - full[:n])
        heat = 1024 * (size[2] + 2 * size[1] ** 2) / t**2
        assert np.all(np.delete(off, 4, axis=1) <= levels * 2.0**-50 * np.delete(size, 4))
        assert np.all(off[:, 4] <= levels * 2.0**-50 * heat)
