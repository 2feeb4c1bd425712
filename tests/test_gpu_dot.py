"""Dot and norm on a GB300 against exact sums, at the edges of the dot's blocks (one
block to 2,048 merged entries, two, four and eight entries a thread to 77,824,
155,648 and beyond, a separate sum above 608 blocks).  Products and their sums are
kept in twice the working precision within a block, the blocks' sums are rounded,
and so is their sum: at most 3 * 2^-53 of the sum of magnitudes.  The norm is the
root of such a sum."""
import math
from fractions import Fraction

import numpy as np
import pytest

import sfci_gb300 as sg
from sfci_gb300 import fcidump as fd

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def contexts(tmp_path_factory):
    d = tmp_path_factory.mktemp("in")
    out = {}
    for words, M in ((1, 28), (2, 34)):
        path = str(d / ("m%d_IN" % M))
        fd.rhf_to_in_file(path, M, 4, 3)
        out[words] = sg.Context(path, 2 * M, 4, Nd=10)
    return out


def wide(keys, words):
    return keys if words == 1 else np.stack([keys, np.zeros(len(keys), np.uint64)], 1)


@pytest.mark.parametrize("words", [1, 2])
@pytest.mark.parametrize("na,nb", [(1, 1), (300, 5), (1024, 1024), (1025, 1024), (38912, 38912), (38913, 38912),
                                   (77824, 77825), (900000, 400001)])
def test_dot_and_norm(contexts, words, na, nb):
    c = contexts[words]
    rng = np.random.default_rng([na, nb, words])
    pool = np.unique(rng.integers(0, 1 << 54, na + nb + 1000, dtype=np.uint64))
    ka = np.sort(rng.choice(pool, na, replace=False))
    both = rng.choice(ka, min(na, nb) * 2 // 3 + 1, replace=False)[:nb]
    rest = np.setdiff1d(pool, ka)
    kb = np.sort(np.concatenate([both, rng.choice(rest, nb - len(both), replace=False)]))
    aa, ab = (rng.standard_normal(n) * np.exp(rng.uniform(-20, 20, n)) for n in (na, nb))
    v, w = c.vec_from(wide(ka, words), aa), c.vec_from(wide(kb, words), ab)
    common, ia, ib = np.intersect1d(ka, kb, return_indices=True)
    prods = [Fraction(float(x)) * Fraction(float(y)) for x, y in zip(aa[ia], ab[ib])]
    exact, mag = sum(prods), sum(abs(p) for p in prods)
    got = v.dot(w)
    assert abs(Fraction(got) - exact) <= 3 * mag / 2 ** 53
    assert all(v.dot(w) == got for _ in range(5))
    # the squares of na entries, and a root: half an ulp of the sum and one of the root
    sq = sum(Fraction(float(x)) ** 2 for x in aa)
    n = v.norm()
    if na <= 1 << 20:
        assert abs(Fraction(n) ** 2 - sq) <= 6 * sq / 2 ** 53


@pytest.mark.parametrize("words", [1, 2])
def test_repeated_keys_match_every_time(contexts, words):
    """An entry of the second vector meets the first one's key as often as it repeats."""
    c = contexts[words]
    ka = np.arange(100, dtype=np.uint64) * np.uint64(3)
    kb = np.sort(np.concatenate([ka[5:90], np.repeat(ka[10:12], 11)]))
    aa, ab = np.arange(100) + 1.0, np.ones(len(kb))
    v, w = c.vec_from(wide(ka, words), aa), c.vec_from(wide(kb, words), ab)
    assert v.dot(w) == sum(aa[int(k) // 3] for k in kb)


@pytest.mark.parametrize("x", [math.inf, -math.inf, math.nan])
def test_values_that_are_not_finite(contexts, x):
    c = contexts[1]
    k = np.arange(5000, dtype=np.uint64)
    a = np.ones(5000)
    a[1234] = x
    v, w = c.vec_from(k, a), c.vec_from(k, np.full(5000, 2.0))
    assert v.dot(w) == x if x == x else v.dot(w) != v.dot(w)
    assert v.norm() == math.inf if x == x else v.norm() != v.norm()
