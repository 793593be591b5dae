"""Ising bins whose edges are no energies (energy_min off the grid of 4 |J|): the general kernel takes them, whatever the
lattice size, bit for bit with the oracle."""
import pytest

from test_gpu_parity import _compare, _pair


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [-2.0, -1.0, 1.0])
@pytest.mark.parametrize("L", [8, 16, 20, 24, 32])
def test_energy_min_off_the_grid(engine_lib, oracle_lib, L, offset):
    N = L * L
    eng, orc = _pair(engine_lib, oracle_lib, 0, L, -2.0 * N + offset, 2.0 * N + offset + 4, 4.0, 3, 2, 8, 16, 5 + L)
    try:
        assert eng.launch_shapes()[0][1] == 0                  # not the bin-tracking kernel
        for k in range(2):
            eng.run_cycles(1)
            orc.cycle()
            _compare(eng, orc, f"cycle {k}")
    finally:
        eng.close()
        orc.close()
