"""Which route the energy and the linear product's dots take on a GB300, and that
both give the same.  The energy's statistics count the neighbouring alpha strings
of the pair search; a projection by pair search makes at least 22 launches (two rank
passes of three, two lists of five, two neighbour passes, a scan, diagonals, an
offset copy, the search), by sweep at most 7 (diagonals, scan of up to three, sweep),
and 17 others are common to both (table, at most 3 insertions, 6 for the dots, 7 for
the sums of three vectors)."""
import numpy as np
import pytest

import sfci_gb300 as sg
from sfci_gb300 import fcidump as fd
from test_gpu_pairs import CASES, system
from test_gpu_rows import vector

pytestmark = pytest.mark.gpu

SEARCH = {"small strings", "unequal spins", "oriented alpha-beta integrals", "32 orbitals of a spin", "two-word keys",
          "one electron of a spin", "one hole of a spin"}


@pytest.mark.parametrize("name", list(CASES))
def test_energy_route(name, tmp_path):
    M, kind, na, nb, n = CASES[name]
    path = system(tmp_path, M, kind, na + nb)
    keys, amps = vector(M, na, nb, n, np.random.default_rng(19))
    c = sg.Context(path, 2 * M, na + nb, Nd=n)
    c.calc_energy(c.vec_from(keys, amps))
    assert (c.last_stats()["leaves"] > 0) == (name in SEARCH), c.last_stats()


@pytest.mark.parametrize("M,n", [(14, 2500), (34, 1303)])
def test_a_device_budget_bounds_the_pair_search(M, n, tmp_path):
    """The search of these vectors takes more than the 32 bytes a determinant of its
    lists; a budget of those goes to the sweep, whose sums round each product and
    partial sum once more: 1e-13 as in test_gpu_pairs."""
    path = str(tmp_path / "sys_IN")
    fd.rhf_to_in_file(path, M, 10, 3)
    keys, amps = vector(M, 5, 5, n, np.random.default_rng(31))
    got = []
    for budget in (0, 64 << 30, 32 * n):
        c = sg.Context(path, 2 * M, 10, Nd=n, mem_budget=budget)
        e = c.calc_energy(c.vec_from(keys, amps))
        got.append((e, c.last_stats()["leaves"]))
    assert got[0] == got[1] and got[0][1] > 0 and got[2][1] == 0
    assert abs(got[2][0] - got[0][0]) < 1e-13


def test_projection_route(tmp_path):
    path = str(tmp_path / "sys_IN")
    fd.rhf_to_in_file(path, 14, 10, 3)
    keys, amps = vector(14, 5, 5, 2500, np.random.default_rng(31))
    c = sg.Context(path, 28, 10, Nd=2500, mem_budget=64 << 30)
    v, out = c.vec_from(keys, amps), c.vec(400000)
    vecs = [c.vec_from(keys[::2], amps[::2]), c.vec_from(keys[1::2], amps[1::2]), v]
    made = []
    for f in (lambda: c.SpMVMtply_bucket(v, out, 0.5, 1.0), lambda: c.spmspvm_bucket_linear(v, out, 0.5, vecs)):
        f()
        n = c.launches()
        f()
        made.append(c.launches() - n)
    assert made[1] - made[0] > 24


def test_a_full_space_takes_the_sweep(tmp_path):
    """Every determinant of 20 spin orbitals with 5 electrons a spin: each would be
    compared with 6,552 others for its 1,126 terms, more than the search's limit of
    four a term.  Bounds on the energy as in test_gpu_pairs."""
    from itertools import combinations
    path = system(tmp_path, 10, "rhf", 10)
    s = [sum(1 << 2 * i for i in o) for o in combinations(range(10), 5)]
    keys = np.sort(np.array([a | b << 1 for a in s for b in s], np.uint64))
    amps = np.random.default_rng(37).standard_normal(len(keys))
    amps /= np.linalg.norm(amps)
    c = sg.Context(path, 20, 10, Nd=len(keys), coeff_cut=-1.0)
    v, out = c.vec_from(keys, amps), c.vec(len(keys))
    d = c.SpMVMtply_bucket(v, out, 0.0, 1.0)
    assert abs(c.calc_energy(v) - d) < 1e-13 and c.last_stats()["leaves"] == 0


@pytest.mark.parametrize("M,n,B,search", [(28, 64, 20000, False), (28, 1000, 1000, True), (34, 300, 20000, False)])
def test_a_short_vector_on_a_long_basis_takes_the_sweep(M, n, B, search, tmp_path):
    """1.2e6 terms against 65,536 slots, 1.8e7 against 2,048, 8.8e6 against 65,536 with
    280,000 strings of a spin.  The dot with the basis whole and in two halves is the
    same sum but for its additions: at most 30 roundings in a row (a thread's few and
    two trees of 256), of partial sums below |v| |H| = 100, 3.4e-13."""
    path = str(tmp_path / "sys_IN")
    fd.rhf_to_in_file(path, M, 10, 3)
    rng = np.random.default_rng(41)
    keys, amps = vector(M, 5, 5, n, rng)
    kb, ab = vector(M, 5, 5, B, rng)
    c = sg.Context(path, 2 * M, 10, Nd=n, mem_budget=64 << 30)
    v, out, b = c.vec_from(keys, amps), c.vec(400000), c.vec_from(kb, ab)
    made = []
    for f in (lambda: c.SpMVMtply_bucket(v, out, 0.5, 1.0), lambda: c.spmspvm_bucket_linear(v, out, 0.5, [b])):
        f()
        k = c.launches()
        f()
        made.append(c.launches() - k)
    assert (made[1] - made[0] > 24) == search
    whole = c.spmspvm_bucket_linear(v, out, 0.5, [b])
    parts = c.spmspvm_bucket_linear(v, out, 0.5, [c.vec_from(kb[::2], ab[::2]), c.vec_from(kb[1::2], ab[1::2])])
    assert abs(whole[0] - parts.sum()) <= 1e-12
