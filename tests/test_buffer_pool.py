"""The device and pinned buffer pools over a driver that counts and runs out:
spare buffers never make another allocation fail, a pool keeps its limit, and
nothing is released twice or lost, from one thread or several."""
import ctypes as C
import os
import subprocess

import pytest

from beep_gb300 import build as bb

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("pool") / "pool.so")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(bb.nvcc()))), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-pthread", "-I", bb.CSRC, "-I", cuda,
                    os.path.join(HERE, "buffer_pool.cc"), "-o", so, "-Wl,-Bsymbolic"], check=True)
    return C.CDLL(so)


@pytest.mark.parametrize("case", ["spare_of_other_pools_is_given_up", "a_failed_allocation_leaves_nothing_behind",
                                  "a_pool_keeps_its_limit_and_trims_the_oldest",
                                  "large_buffers_take_what_they_ask_for", "threads_share_pools_of_a_full_device"])
def test_pools(lib, case):
    assert getattr(lib, case)() == 0
