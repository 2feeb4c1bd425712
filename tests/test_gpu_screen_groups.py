"""The number of a vector's screened groups on a GB300: counted without the network
it is the number that a prediction reports, and the sum of the groups of each
determinant, C(n,2) (v-1) a spin and n_a v_a n_b over both (n electrons, v holes)."""
from math import comb

import numpy as np
import pytest

import sfci_gb300 as sg
from sfci_gb300 import fcidump as fd
from test_gpu_rows import vector

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,na,nb,n", [(14, 5, 5, 1), (14, 4, 6, 333), (34, 3, 5, 257)])
def test_group_count(M, na, nb, n, tmp_path):
    path = str(tmp_path / "sys_IN")
    fd.rhf_to_in_file(path, M, na + nb, 3)
    keys, amps = vector(M, na, nb, n, np.random.default_rng(61))
    c = sg.Context(path, 2 * M, na + nb, Nd=n)
    v, s = c.vec_from(keys, amps), sg.Screen(c, seed=1)
    per = comb(na, 2) * (M - na - 1) + comb(nb, 2) * (M - nb - 1) + na * (M - na) * nb
    p = s.predict(v, 0.5, probs=True)
    assert s.groups_of(v) == p["groups"] == len(p["prob"]) == n * per
