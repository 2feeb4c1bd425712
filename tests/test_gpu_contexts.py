"""Several contexts at work at once on a GB300, each on a thread of its own: the key
sort and the selection wait for their whole grid while another context's long
kernels hold the SMs, and products of different systems launch the same kernels
with different shared-memory sizes.  Every result is the one the context gives
alone."""
import threading

import numpy as np
import pytest

import sfci_gb300 as sg
from sfci_gb300 import fcidump as fd
from test_gpu_prims import distinct_keys
from test_gpu_rows import vector

pytestmark = pytest.mark.gpu


def run_together(jobs):
    errors = []

    def guard(job):
        try:
            job()
        except BaseException as e:  # a failed assertion or an error status
            errors.append(repr(e))

    threads = [threading.Thread(target=guard, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_sorts_and_selections_beside_long_products(tmp_path):
    path = str(tmp_path / "sys_IN")
    fd.rhf_to_in_file(path, 28, 8, 3)
    rng = np.random.default_rng(17)
    keys, amps = vector(28, 4, 4, 60000, rng)
    busy = sg.Context(path, 56, 8, Nd=60000)
    v, out = busy.vec_from(keys, amps), busy.vec(2000000)
    stop = threading.Event()

    def products():
        try:
            first = busy.SpMVMtply_bucket(v, out, 0.0, 1.0)
            for _ in range(12):
                assert busy.SpMVMtply_bucket(v, out, 0.0, 1.0) == first
        finally:
            stop.set()

    def sorts(seed):
        def job():
            r = np.random.default_rng(seed)
            n = 700001
            k, a = distinct_keys(n, 1, 56, r), r.standard_normal(n)
            order = np.argsort(k)
            big = np.sort(np.argsort(np.abs(a[order]), kind="stable")[n - n // 3:])
            c = sg.Context(path, 56, 8, Nd=10)
            x, y = c.vec(n), c.vec(n // 3)
            while True:
                last = stop.is_set()
                x.upload(k, a)
                y.shrinkFrom(x)
                kk, aa = y.download()
                assert np.array_equal(kk, k[order][big]) and np.array_equal(aa, a[order][big])
                if last:
                    return
        return job

    run_together([products, sorts(1), sorts(2)])


def test_products_of_systems_of_different_sizes(tmp_path):
    """The row kernels take 7 words a single excitation of shared memory besides their
    tables: 45, 115 and 48 of them here.  (A launch that found another thread's
    smaller limit failed with an invalid value; the window is short, so a run without
    an error proves little, one with an error all.)"""
    def job(M, na, n, seed):
        path = str(tmp_path / ("m%d_IN" % M))
        fd.rhf_to_in_file(path, M, 2 * na, 3)
        keys, amps = vector(M, na, na, n, np.random.default_rng(seed))

        def run():
            c = sg.Context(path, 2 * M, 2 * na, Nd=n)
            v, out = c.vec_from(keys, amps), c.vec(100000)
            first = c.SpMVMtply_bucket(v, out, 0.0, 1.0)
            k, a = out.download()
            for _ in range(100):
                assert c.SpMVMtply_bucket(v, out, 0.0, 1.0) == first
            k1, a1 = out.download()
            assert np.array_equal(k, k1) and np.array_equal(a, a1)
        return run

    run_together([job(14, 5, 2500, 1), job(28, 5, 1000, 2), job(16, 4, 2000, 3)])
