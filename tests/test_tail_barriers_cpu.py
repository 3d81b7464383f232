"""The named barriers of the dense tail's factorisation (tail_barriers.hpp),
run by a CPU model in every order in which the lead and the six other warps can
come to them, for every size of the tail (at most 18 scalars): all orders end,
and no column is used before it is complete. The model itself is checked with
all columns published at one barrier, where a late warp is left behind. No
GPU."""
import ctypes as C
import glob
import os
import re
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


def test_warps_come_to_named_barriers_whole():
    """The named barriers of the kernels are the form that takes a warp as a
    whole: each is written directly behind a warp barrier."""
    found = 0
    for path in sorted(glob.glob(os.path.join(ROOT, "kimera-rpgo_gb300", "csrc", "*.cu*"))):
        lines = [x.strip() for x in open(path) if x.strip() and not x.strip().startswith("//")]
        for k, line in enumerate(lines):
            if re.search(r'"bar\.(sync|arrive|red)', line):
                found += 1
                assert lines[k - 1] == "__syncwarp();", f"{os.path.basename(path)}: {line}"
    assert found >= 4
