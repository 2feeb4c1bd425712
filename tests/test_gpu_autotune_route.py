"""The autotuner on an ordinary context of a GB300: its plans shape the partitioned
product, so that is what it times, also where the row form takes plain products.
The last candidate timed leaves its statistics: a power of two of leaves, as in a
context with a device budget, and not the row form's work units."""
import numpy as np
import pytest

import sfci_gb300 as sg
from sfci_gb300 import fcidump as fd
from test_gpu_rows import vector

pytestmark = pytest.mark.gpu


def test_autotune_times_the_partitioned_product(tmp_path):
    path = str(tmp_path / "sys_IN")
    fd.rhf_to_in_file(path, 14, 10, 3)
    keys, amps = vector(14, 5, 5, 2500, np.random.default_rng(43))
    got = []
    for budget in (0, 64 << 30):
        c = sg.Context(path, 28, 10, Nd=2500, mem_budget=budget)
        v, out = c.vec_from(keys, amps), c.vec(400000)
        c.autotune(v, out)
        tuned = c.last_stats()["leaves"]
        d = c.SpMVMtply_bucket(v, out, 0.0, 1.0)
        got.append((tuned, c.last_stats()["leaves"], d, *out.download()))
    (t0, p0, d0, k0, a0), (t1, p1, d1, k1, a1) = got
    assert t0 == t1 and t0 & (t0 - 1) == 0
    assert p0 != p1  # the product after it: the row form again, and the pipeline
    assert d0 == d1 and np.array_equal(k0, k1) and np.array_equal(a0.view(np.uint64), a1.view(np.uint64))
