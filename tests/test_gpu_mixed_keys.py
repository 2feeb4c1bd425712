"""Vectors that the row form and the pair search decline by their keys (mixed spin
counts, a repeated determinant), on a GB300: one launch finds them, before any
table is built (split, diagonals, marks and two scans: at least five), and the calls
give what the partitioned pipeline and the sweep give.  The pipeline's own plan may
differ by a launch or two between the two contexts, whose memory differs."""
import numpy as np
import pytest

import sfci_gb300 as sg
from sfci_gb300 import fcidump as fd
from test_gpu_rows import vector

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [14, 34])
@pytest.mark.parametrize("what", ["mixed", "twice", "last differs"])
def test_other_keys_cost_one_launch(M, what, tmp_path):
    path = str(tmp_path / "sys_IN")
    fd.rhf_to_in_file(path, M, 10, 3)
    rng = np.random.default_rng(71)
    keys, amps = vector(M, 5, 5, 2500, rng)
    if what == "twice":
        keys, amps = np.concatenate([keys, keys[-1:]]), np.concatenate([amps, amps[-1:]])
    else:
        n = 1500 if what == "mixed" else 1
        k2, a2 = vector(M, 4, 6, n, rng)
        keys, amps = np.concatenate([keys, k2]), np.concatenate([amps, a2])
    got = []
    for budget in (0, 64 << 30):
        c = sg.Context(path, 2 * M, 10, Nd=len(amps), mem_budget=budget)
        v, out = c.vec_from(keys, amps), c.vec(400000)
        c.SpMVMtply_bucket(v, out, 0.5, 1.0)
        for _ in range(2):  # the second time the check's flag has been set before
            n = c.launches()
            d = c.SpMVMtply_bucket(v, out, 0.5, 1.0)
            n = c.launches() - n
        got.append((n, d, *out.download()))
        if not budget:
            l0 = c.launches()
            e = c.calc_energy(v)
            assert c.last_stats()["leaves"] == 0 and c.launches() - l0 <= 10  # check, diagonals, scan, table, sweep, sum
            good = c.vec_from(*vector(M, 5, 5, 2500, np.random.default_rng(72)))
            c.calc_energy(good)
            assert c.last_stats()["leaves"] > 0  # the next vector is searched again
            c.calc_energy(v)
    (n, d, k, a), (n0, d0, k0, a0) = got
    assert n - n0 < 5 and d == d0
    assert np.array_equal(k, k0) and np.array_equal(a.view(np.uint64), a0.view(np.uint64))
