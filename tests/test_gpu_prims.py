"""Key sort and magnitude selection on a GB300 through the vector calls, at the
edges of their warps, slices and of the single-launch sort (6,291,456 entries):
keys and amplitudes must come out exactly as numpy's stable sorts give them."""
import numpy as np
import pytest

import sfci_gb300 as sg
from sfci_gb300 import fcidump as fd

pytestmark = pytest.mark.gpu

SIZES = [2, 31, 33, 1023, 1024, 1025, 5000, 152 * 1024, 152 * 1024 + 1, 700001, (6 << 20) + 1]


@pytest.fixture(scope="module")
def contexts(tmp_path_factory):
    d = tmp_path_factory.mktemp("in")
    out = {}
    for words, M in ((1, 28), (2, 34)):
        path = str(d / ("m%d_IN" % M))
        fd.rhf_to_in_file(path, M, 8, 3) if M == 28 else fd.rhf_to_in_file(path, M, 4, 3)
        out[words] = sg.Context(path, 2 * M, 8 if M == 28 else 4, Nd=10)
    return out


def distinct_keys(n, words, bits, rng):
    lo = np.unique(rng.integers(0, 1 << min(bits, 62), 2 * n + 64, dtype=np.uint64))
    lo = rng.permutation(lo)[:n]
    if words == 1:
        return lo
    return np.stack([lo * np.uint64(4) + np.uint64(1), rng.integers(0, 1 << (bits - 64), n, dtype=np.uint64)], 1)


@pytest.mark.parametrize("words", [1, 2])
@pytest.mark.parametrize("n", SIZES)
def test_unsorted_upload_is_sorted_by_key(contexts, n, words):
    rng = np.random.default_rng(n)
    keys = distinct_keys(n, words, 56 if words == 1 else 68, rng)
    amps = rng.standard_normal(n)
    k, a = contexts[words].vec_from(keys, amps).download()
    order = np.argsort(keys) if words == 1 else np.lexsort((keys[:, 0], keys[:, 1]))
    assert np.array_equal(k, keys[order]) and np.array_equal(a, amps[order])


def values(kind, n, rng):
    if kind == "spread":
        return rng.standard_normal(n) * np.exp(-rng.uniform(0, 30, n))
    if kind == "ties":
        return rng.choice([0.0, -0.0, 1e-3, -1e-3, 2.5, -2.5, 5e-324, np.inf], n)
    return np.full(n, -0.125)  # all equal


@pytest.mark.parametrize("kind", ["spread", "ties", "equal"])
@pytest.mark.parametrize("n", SIZES)
def test_selection_keeps_the_largest_and_the_highest_tied_keys(contexts, n, kind):
    rng = np.random.default_rng(n + 1)
    c = contexts[1]
    keys = np.sort(distinct_keys(n, 1, 56, rng))
    amps = values(kind, n, rng)
    v = c.vec_from(keys, amps)
    for k in sorted({1, n // 3, n // 2, n - 1, n} - {0}):
        w = c.vec(k)
        w.shrinkFrom(v)
        kk, aa = w.download()
        order = np.argsort(np.abs(amps), kind="stable")  # ascending: of equal ones the later keys last
        sel = np.sort(order[n - k:])
        assert np.array_equal(kk, keys[sel])
        assert np.array_equal(aa.view(np.uint64), amps[sel].view(np.uint64))


@pytest.mark.parametrize("n", [1, 40, 3000, 200003])
def test_capped_sum_and_tiny_filter(contexts, n):
    """addThree: x + y + z merged, the Nd largest, entries up to 1e-14 dropped."""
    rng = np.random.default_rng(n + 2)
    c = contexts[1]
    keys = np.sort(distinct_keys(n, 1, 56, rng))
    amps = np.where(rng.random(n) < 0.5, 1e-15, 1.0) * rng.uniform(0.5, 1.0, n)
    v, zero, out = c.vec_from(keys, amps), c.vec(1), c.vec(n)
    for nd in (n, max(1, n // 2)):
        c.set_Nd(nd)
        out.addThree(v, zero, zero, 1.0, 0.0, 0.0)
        k, a = out.download()
        sel = np.sort(np.argsort(np.abs(amps), kind="stable")[n - nd:])
        sel = sel[np.abs(amps[sel]) > 1e-14]
        assert np.array_equal(k, keys[sel]) and np.array_equal(a, amps[sel])
