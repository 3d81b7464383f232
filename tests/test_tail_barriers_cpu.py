"""The named barriers of the dense tail's factorisation (tail_barriers.hpp),
run by a CPU model in every order in which the lead and the six other warps can
come to them, for every size of the tail (at most 18 scalars): all orders end,
and no column is used before it is complete. The model itself is checked with
all columns published at one barrier, where a late warp is left behind. No
GPU."""
import ctypes as C
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("tb") / "libtailbarriers.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "kimera-rpgo_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "tail_barriers.cpp"), "-o", out], check=True)
    return C.CDLL(out)


@pytest.mark.parametrize("n", [3, 6, 9, 12, 15, 18])
def test_every_order_ends(lib, n):
    states = C.c_int64(0)
    assert lib.tail_barriers_check(n, 7, 0, C.byref(states)) == 0
    assert states.value > 100 * n


@pytest.mark.parametrize("n", [3, 18])
def test_one_barrier_leaves_a_late_warp_behind(lib, n):
    assert lib.tail_barriers_check(n, 7, 1, C.byref(C.c_int64(0))) == 1
