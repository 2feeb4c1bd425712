"""Energy and projection by the pair search (pairs.cu) on a GB300.

calc_energy rounds each product c_q (c_p H_qp) twice and sums exactly; <v|Hv> of
the partitioned product rounds each product c_q (H v)_q once and sums exactly.
They differ by at most 3 * 2^-53 * sum |c_q H_qp c_p|, and |H| has row sums below
100 for these systems (a diagonal below 40 and at most 62,000 elements of 1e-3), so
by less than 1e-13 for a normalised vector.  The dots <basis_j | (H - lambda) v>
are exact sums rounded once, multiplied and added in 64 bits: 1e-12 of the sum of
magnitudes bounds n additions of n < 4,000 products."""
import numpy as np
import pytest

import sfci_gb300 as sg
from sfci_gb300 import fcidump as fd
from test_gpu_rows import vector

pytestmark = pytest.mark.gpu

# spatial orbitals, integrals, alpha and beta electrons, determinants
CASES = {"small strings": (10, "rhf", 5, 5, 3000), "few": (14, "rhf", 5, 5, 65), "unequal spins": (12, "rhf", 3, 6, 2000),
         "one electron of a spin": (20, "rhf", 1, 6, 2500), "one hole of a spin": (16, "rhf", 15, 5, 1500),
         "oriented alpha-beta integrals": (14, "uhf", 6, 6, 1501), "32 orbitals of a spin": (32, "rhf", 4, 5, 2001),
         "two-word keys": (34, "rhf", 5, 5, 1303)}


def system(tmp_path, M, kind, ne):
    path = str(tmp_path / "sys_IN")
    if kind == "rhf":
        fd.rhf_to_in_file(path, M, ne, 3)
    else:
        fd.uhf_to_in_file(path, M, ne, 2, 3)
    return path


def lookup(keys, amps, of):
    """Amplitudes of the keys `of` in a vector with ascending keys."""
    def ordered(k):
        k = k.reshape(len(k), -1)
        r = np.zeros(len(k), [("hi", "u8"), ("lo", "u8")])
        r["lo"], r["hi"] = k[:, 0], k[:, 1] if k.shape[1] == 2 else 0
        return r
    have, want = ordered(keys), ordered(of)
    i = np.minimum(np.searchsorted(have, want), len(have) - 1)
    return np.where(have[i] == want, amps[i], 0.0)


@pytest.mark.parametrize("name", list(CASES))
def test_energy_and_projection(name, tmp_path):
    M, kind, na, nb, n = CASES[name]
    path = system(tmp_path, M, kind, na + nb)
    rng = np.random.default_rng(19)
    keys, amps = vector(M, na, nb, n, rng)
    c = sg.Context(path, 2 * M, na + nb, Nd=n, coeff_cut=-1.0, mem_budget=64 << 30)
    v, out = c.vec_from(keys, amps), c.vec(40000000)
    d = c.SpMVMtply_bucket(v, out, 0.0, 1.0)
    assert abs(c.calc_energy(v) - d) < 1e-13
    # basis: subsets of the vector's own support with other amplitudes, and the vector
    lam = -1.25
    c.SpMVMtply_bucket(v, out, lam, 1.0)
    basis = []
    for frac in (0.3, 1.0):
        sel = np.sort(rng.choice(n, max(2, int(frac * n)), replace=False))
        basis.append((keys[sel], rng.standard_normal(len(sel))))
    basis.append((keys, amps))
    vecs = [c.vec_from(k, a) for k, a in basis]
    h = c.spmspvm_bucket_linear(v, c.vec(100000), lam, vecs)
    wk, wa = out.download()
    for (k, a), got in zip(basis, h):
        w = lookup(wk, wa, k)
        assert abs(got - np.dot(a, w)) <= 1e-12 * np.sum(np.abs(a * w)), name


def test_energy_of_mixed_spin_counts_takes_the_general_sweep(tmp_path):
    path = system(tmp_path, 14, "rhf", 10)
    rng = np.random.default_rng(23)
    k1, a1 = vector(14, 5, 5, 300, rng)
    k2, a2 = vector(14, 4, 6, 300, rng)
    c = sg.Context(path, 28, 10, Nd=1000)
    e1, e2 = c.calc_energy(c.vec_from(k1, a1)), c.calc_energy(c.vec_from(k2, a2))
    both = c.calc_energy(c.vec_from(np.concatenate([k1, k2]), np.concatenate([a1, a2])))
    assert abs(both - (e1 + e2)) < 1e-12
