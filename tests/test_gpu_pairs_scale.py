"""calc_energy on vectors that are not normalised, on a GB300: <s v|H|s v> is
s^2 <v|H|v>, and for a power of two s every product and every sum is the scaled one
exactly, so the energies agree bit for bit, in the general sweep (65 determinants of
28 spin orbitals, 1.8e5 terms) and in the pair search (2,000 determinants)."""
import numpy as np
import pytest

import sfci_gb300 as sg
from sfci_gb300 import fcidump as fd
from test_gpu_rows import vector

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [14, 34])
@pytest.mark.parametrize("n", [65, 2000])
def test_energy_scales_with_the_vector(M, n, tmp_path):
    path = str(tmp_path / "sys_IN")
    fd.rhf_to_in_file(path, M, 10, 3)
    keys, amps = vector(M, 5, 5, n, np.random.default_rng(5))
    c = sg.Context(path, 2 * M, 10, Nd=n)
    e = c.calc_energy(c.vec_from(keys, amps))
    for k in (-300, -35, -20, 20, 35, 300):
        assert c.calc_energy(c.vec_from(keys, amps * 2.0 ** k)) == e * 4.0 ** k, k


def test_energy_of_vectors_at_the_ends_of_the_range(tmp_path):
    """Zero and subnormal amplitudes give 0; infinities and NaNs a value that is not finite."""
    path = str(tmp_path / "sys_IN")
    fd.rhf_to_in_file(path, 14, 10, 3)
    keys, amps = vector(14, 5, 5, 2000, np.random.default_rng(5))
    c = sg.Context(path, 28, 10, Nd=2000)
    assert c.calc_energy(c.vec_from(keys, 0.0 * amps)) == 0.0
    assert c.calc_energy(c.vec_from(keys, np.full(2000, 5e-324))) == 0.0
    for x in (np.inf, np.nan):
        bad = amps.copy()
        bad[7] = x
        assert not np.isfinite(c.calc_energy(c.vec_from(keys, bad)))
