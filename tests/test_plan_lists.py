"""When the lists that the row product and the pair search keep make way for the
partitioned product's memory plan (csrc/plan.h), on the host."""
import ctypes as C
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "sfci_gb300", "csrc")
GB = 1 << 30


@pytest.fixture(scope="module")
def wants(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("pl") / "lists.so")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-I" + CSRC,
                        os.path.join(ROOT, "tests", "native", "lists_host.cpp"), "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(so)
    L.pl_wants_lists.argtypes = [C.c_uint64] * 6
    return lambda free, held, lists, T, tb=16, budget=0: bool(
        L.pl_wants_lists(int(free), int(held), int(lists), int(T), tb, int(budget)))


def test_lists_stay_beside_a_plan_that_already_holds_its_memory(wants):
    """3e9 terms want 144 GB; the plan holds 180 GB of it, 20 GB are free, the lists
    hold 60: nothing of the plan has to grow."""
    assert not wants(20 * GB, 180 * GB, 60 * GB, 3e9)


def test_lists_make_way_for_a_plan_that_does_not_fit_beside_them(wants):
    assert wants(100 * GB, 0, 150 * GB, 3e9)
    assert wants(20 * GB, 80 * GB, 150 * GB, 3e9)
    assert wants(20 * GB, 180 * GB, 60 * GB, 3e10)


def test_lists_that_would_not_change_the_plan_stay(wants):
    assert not wants(250 * GB, 0, 1 * GB, 3e10)  # too many terms for the GPU, whatever is freed
    assert not wants(250 * GB, 0, 0, 3e10)
    assert not wants(200 * GB, 0, 60 * GB, 1e9)


def test_a_device_budget_bounds_what_the_plan_wants(wants):
    assert not wants(30 * GB, 0, 200 * GB, 3e10, budget=20 * GB)
    assert wants(30 * GB, 0, 200 * GB, 3e10, budget=100 * GB)
