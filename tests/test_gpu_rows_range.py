"""Products whose terms the row form's accumulators do not take (2^15 at these
sizes), on a GB300: the partitioned pipeline's product, bit for bit, and no row form
run in vain before it.  The kernels up to the first readback (split, diagonals, one
mark, two scans of at most three launches) and the partitioned pipeline make at
most 12 launches more than the pipeline alone; the whole row form makes 30."""
import numpy as np
import pytest

import sfci_gb300 as sg
from sfci_gb300 import fcidump as fd
from test_gpu_rows import vector

pytestmark = pytest.mark.gpu


def products(path, M, ne, keys, amps, lam):
    got = []
    for budget in (0, 64 << 30):  # a context with a budget never takes the row form
        c = sg.Context(path, 2 * M, ne, Nd=len(amps), mem_budget=budget)
        v, out = c.vec_from(keys, amps), c.vec(400000)
        c.SpMVMtply_bucket(v, out, lam, 1.0)
        n = c.launches()
        d = c.SpMVMtply_bucket(v, out, lam, 1.0)
        n = c.launches() - n
        got.append((*out.download(), d, n))
    (k, a, d, n), (k0, a0, d0, n0) = got
    assert np.array_equal(k, k0) and np.array_equal(a.view(np.uint64), a0.view(np.uint64)) and d == d0
    return n, n0


@pytest.mark.parametrize("M,n", [(14, 2500), (28, 3001), (34, 1601)])
def test_a_diagonal_term_out_of_range_declines_the_row_form_at_once(M, n, tmp_path):
    path = str(tmp_path / "sys_IN")
    fd.rhf_to_in_file(path, M, 10, 3)
    keys, amps = vector(M, 5, 5, n, np.random.default_rng(3))
    rows, parts = products(path, M, 10, keys, amps * 2.0 ** 17, 0.0)
    assert rows - parts <= 12
    rows, parts = products(path, M, 10, keys, amps, 0.0)  # in range: the row form itself
    assert rows != parts


def test_an_off_diagonal_term_out_of_range_ends_the_rows(tmp_path):
    path = str(tmp_path / "sys_IN")
    fd.rhf_to_in_file(path, 28, 10, 3)
    keys, amps = vector(28, 5, 5, 3001, np.random.default_rng(3))
    amps = amps / np.abs(amps).max() * 1e-3
    amps[0] = 2.0 ** 22  # its diagonal term is zero; elements of 2^-7 and more are out of range, all are below 2
    c = sg.Context(path, 56, 10)
    products(path, 28, 10, keys, amps, float(c.DiagCal_bit(keys[:1])[0]))
