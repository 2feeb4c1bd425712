"""Energies in spaces so full that the sweep is faster than the pair search, on a
GB300: the call makes the sweep's launches and a first readback of the key, and
not the search's lists (at least 14 launches: two rank kernels and a scan, two list
passes with scans, a neighbour pass with a scan, diagonals)."""
from itertools import combinations

import numpy as np
import pytest

import sfci_gb300 as sg
from sfci_gb300 import fcidump as fd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,na,nb,share", [(16, 15, 5, 0.11), (10, 5, 5, 1.0), (12, 11, 6, 0.3)])
def test_full_spaces_decline_before_the_lists(M, na, nb, share, tmp_path):
    path = str(tmp_path / "sys_IN")
    fd.rhf_to_in_file(path, M, na + nb, 3)
    s = [[sum(1 << 2 * i for i in o) for o in combinations(range(M), n)] for n in (na, nb)]
    keys = np.array([a | b << 1 for a in s[0] for b in s[1]], np.uint64)
    rng = np.random.default_rng(67)
    keys = np.sort(rng.choice(keys, int(share * len(keys)), replace=False))
    amps = rng.standard_normal(len(keys))
    amps /= np.linalg.norm(amps)
    made = []
    for budget in (0, 1):  # a budget of one byte: the sweep, whatever the space
        c = sg.Context(path, 2 * M, na + nb, Nd=len(keys), mem_budget=budget)
        v = c.vec_from(keys, amps)
        e = c.calc_energy(v)
        n = c.launches()
        assert c.calc_energy(v) == e
        made.append((c.launches() - n, e))
    assert made[0] == made[1]
