"""The row product keeps its lists between calls; an allocation that finds no room
gets theirs.  A system with 2.8e7 strings of a spin keeps about a gigabyte of them;
a vector fills the device up to 256 MB, and one of 768 MB then takes the lists'
place.  The product still gives what it gave."""
import gc

import numpy as np
import pytest
import torch

import sfci_gb300 as sg
from sfci_gb300 import fcidump as fd
from test_gpu_rows import vector

pytestmark = pytest.mark.gpu


def test_lists_make_way_for_a_vector(tmp_path):
    path = str(tmp_path / "sys_IN")
    fd.rhf_to_in_file(path, 32, 18, 3)
    keys, amps = vector(32, 9, 9, 1500, np.random.default_rng(29))
    c = sg.Context(path, 64, 18, Nd=1500)
    v, out = c.vec_from(keys, amps), c.vec(100000)
    d = c.SpMVMtply_bucket(v, out, 0.0, 1.0)
    before = out.download()
    gc.collect()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    fill = c.vec((free - (256 << 20)) // 16)
    w = c.vec((768 << 20) // 16)
    w.naiveCopy(out)
    assert np.array_equal(w.download()[0], before[0])
    del fill, w
    gc.collect()
    assert c.SpMVMtply_bucket(v, out, 0.0, 1.0) == d
    after = out.download()
    assert np.array_equal(before[0], after[0]) and np.array_equal(before[1], after[1])
