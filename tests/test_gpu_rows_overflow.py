"""Row products whose survivors outgrow their buffer, on a GB300: the buffer is cut
to the output's capacity and the rows left over go on, in several rounds.  Keys,
amplitudes, <v|Hv> and the distinct count are the partitioned pipeline's, bit for
bit.  The overrun allowed to a round is 152 x 10,240 entries, so a small margin gives
about a round for every 1.6 million survivors."""
import numpy as np
import pytest

import sfci_gb300 as sg
from sfci_gb300 import fcidump as fd
from test_gpu_rows import vector

pytestmark = pytest.mark.gpu

# spatial orbitals, integrals, alpha and beta electrons, sources, capacity, margin
CASES = {"large rows": (14, "uhf", 6, 6, 3000, 5000, 1000), "many light rows": (32, "rhf", 4, 5, 3001, 20000, 100000),
         "two-word keys": (34, "rhf", 5, 5, 1601, 20000, 1), "more than 2^15 connections": (34, "rhf", 8, 8, 1201, 20000, 1000000)}


def write(path, M, kind, ne):
    if kind == "rhf":
        fd.rhf_to_in_file(path, M, ne, 3)
    else:
        fd.uhf_to_in_file(path, M, ne, 2, 3)


@pytest.mark.parametrize("name", list(CASES))
def test_rounds_give_the_same_product(name, tmp_path):
    M, kind, na, nb, n, cap, margin = CASES[name]
    path = str(tmp_path / "sys_IN")
    write(path, M, kind, na + nb)
    keys, amps = vector(M, na, nb, n, np.random.default_rng(47))
    got = []
    for budget in (0, 64 << 30):
        c = sg.Context(path, 2 * M, na + nb, Nd=n, coeff_cut=-1.0, mem_budget=budget)
        c.set_row_margin(margin)
        v, out = c.vec_from(keys, amps), c.vec(cap)
        d = c.SpMVMtply_bucket(v, out, 0.5, 1.0)
        got.append((*out.download(), d, c.last_stats()))
    (k, a, d, st), (k0, a0, d0, st0) = got
    assert st["passes"] > 1 and st["leaves"] != st0["leaves"], st
    assert np.array_equal(k, k0) and np.array_equal(a.view(np.uint64), a0.view(np.uint64)) and d == d0
    assert (st["terms"], st["unique"], st["out_len"]) == (st0["terms"], st0["unique"], st0["out_len"])


@pytest.mark.parametrize("M,n", [(28, 1200), (34, 1601)])
def test_rounds_with_extra_sources(M, n, tmp_path):
    path = str(tmp_path / "sys_IN")
    write(path, M, "rhf", 10)
    rng = np.random.default_rng(53)
    keys, amps = vector(M, 5, 5, n, rng)
    kb, ab = vector(M, 5, 5, 5000, rng)
    got = []
    for margin, budget in ((1000, 0), (0, 0), (0, 64 << 30)):
        c = sg.Context(path, 2 * M, 10, Nd=n, coeff_cut=-1.0, mem_budget=budget)
        c.set_row_margin(margin)
        v, out, b = c.vec_from(keys, amps), c.vec(30000), c.vec_from(kb, ab)
        h = c.spmspvm_bucket_linear(v, out, 0.5, [b, v])
        got.append((*out.download(), h, c.last_stats()))
    assert got[0][3]["passes"] > 1 and got[1][3]["passes"] == 1
    for k, a, h, st in got[1:]:
        assert np.array_equal(got[0][0], k) and np.array_equal(got[0][1].view(np.uint64), a.view(np.uint64))
        assert np.array_equal(got[0][2], h) and st["unique"] == got[0][3]["unique"]
