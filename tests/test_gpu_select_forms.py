"""The one-launch sort and selection against the multi-launch forms on a GB300: a
context with the grid barrier switched off takes the chain of launches, and every
call gives the same keys and the same amplitude bits.  Amplitudes hold ties,
signed zeros, infinities and NaNs (of the largest magnitude of all); sizes are the
edges of warps, slices and sort passes."""
import numpy as np
import pytest

import sfci_gb300 as sg
from sfci_gb300 import fcidump as fd
from test_gpu_prims import distinct_keys
from test_gpu_rows import vector

pytestmark = pytest.mark.gpu

SIZES = [2, 33, 1025, 152 * 1024 + 1, 700001]


@pytest.fixture(scope="module")
def contexts(tmp_path_factory):
    """(with, without the barrier) by key words."""
    d = tmp_path_factory.mktemp("in")
    out = {}
    for words, M in ((1, 28), (2, 34)):
        path = str(d / ("m%d_IN" % M))
        fd.rhf_to_in_file(path, M, 4, 3)
        out[words] = [sg.Context(path, 2 * M, 4, Nd=10) for _ in range(2)]
        out[words][1].set_grid_barrier(False)
    return out


def bits(v):
    k, a = v.download()
    return k, a.view(np.uint64)


def same(x, y):
    return np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1])


@pytest.mark.parametrize("words", [1, 2])
@pytest.mark.parametrize("n", SIZES)
def test_sort_and_selection(contexts, n, words):
    rng = np.random.default_rng([n, words])
    keys = distinct_keys(n, words, 56 if words == 1 else 68, rng)
    amps = rng.choice([0.0, -0.0, 1e-3, -1e-3, 2.5, -2.5, 5e-324, np.inf, -np.inf, np.nan, 7.0], n)
    amps[rng.random(n) < 0.4] = rng.standard_normal()
    order = np.argsort(keys) if words == 1 else np.lexsort((keys[:, 0], keys[:, 1]))
    mag = np.abs(amps[order]).view(np.uint64)  # as integers: a NaN is above infinity
    rank = np.argsort(mag, kind="stable")      # ascending: of equal ones the later keys last
    got = []
    for c in contexts[words]:
        l0 = c.launches()
        v = c.vec_from(keys, amps)
        res = [bits(v)]
        for k in sorted({1, n // 3, n - 1} - {0}):
            w = c.vec(k)
            w.shrinkFrom(v)
            res.append(bits(w))
            sel = np.sort(rank[n - k:])
            assert same(res[-1], (keys[order][sel], amps[order][sel].view(np.uint64)))
        c.set_Nd(max(1, n // 2))
        out, zero = c.vec(n), c.vec(1)
        out.addThree(v, zero, zero, 1.0, 0.0, 0.0)  # the largest, less those up to 1e-14
        got.append((res + [bits(out)], c.launches() - l0))
    (x, few), (y, many) = got
    assert few < many
    assert all(same(p, q) for p, q in zip(x, y))


@pytest.mark.parametrize("words", [1, 2])
def test_cut_and_capped_product(contexts, words):
    M = 28 if words == 1 else 34
    keys, amps = vector(M, 2, 2, 900, np.random.default_rng(words))
    got = []
    for c in contexts[words]:
        c.set_Nd(300)  # the product takes the largest 300
        v, empty, r, out = c.vec_from(keys, amps), c.vec(1), c.vec(900), c.vec(1234)
        res = [c.spmspvm_bucket_res_norm(empty, r, v, 0.0), c.SpMVMtply_bucket(v, out, 0.0, 1.0)]
        got.append((res, bits(r), bits(out)))
    (a, ra, oa), (b, rb, ob) = got
    assert a == b and same(ra, rb) and same(oa, ob) and len(oa[0]) == 1234
