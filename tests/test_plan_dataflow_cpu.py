"""The dataflow part of the direct solve's plan (add_dataflow): its products,
row lists and tail entries against the update lists of the level form, over
graph shapes, block sizes and level widths, for single and merged plans
(tests/native/plan_dataflow.cpp). No GPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "kimera-rpgo_gb300", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("df") / "libplandf.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC,
                    os.path.join(ROOT, "tests", "native", "plan_dataflow.cpp"), os.path.join(CSRC, "chol_plan.cpp"),
                    "-lpthread", "-o", out], check=True)
    return C.CDLL(out)


def _graph(shape, n, seed):
    rng = np.random.default_rng(seed)
    if shape == "alone":
        return []
    chain = [(i, i + 1) for i in range(n - 1)]
    if shape == "chain":
        return chain
    if shape == "near":
        return chain + [(i, min(n - 1, i + int(rng.integers(2, 9)))) for i in rng.integers(0, max(n - 3, 1), n // 4)]
    if shape == "tail4":  # a dense tail of four blocks: 24 scalars at d = 6, more entries than threads
        return chain + [(38, 49), (28, 39), (33, 27)]
    if shape == "far":
        return chain + [tuple(int(x) for x in rng.choice(n, 2, replace=False)) for _ in range(n // 5)]
    return chain + [(0, i) for i in range(2, n)]  # a hub: columns beyond the part's limits


@pytest.mark.parametrize("d", [3, 6])
@pytest.mark.parametrize("shape,n", [("alone", 1), ("alone", 5), ("chain", 2), ("chain", 3), ("chain", 70),
                                     ("near", 40), ("near", 700), ("tail4", 50), ("far", 60), ("far", 400), ("hub", 60)])
@pytest.mark.parametrize("cols", [0, 1, 7, 60, 1216])
def test_dataflow_lists_match_the_level_form(lib, d, shape, n, cols):
    e = _graph(shape, n, n)
    kind = np.array([0] * len(e) + [1], np.int32)
    vi = np.array([a for a, _ in e] + [0], np.int32)
    vj = np.array([b for _, b in e] + [0], np.int32)
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)
    info = np.zeros(6, np.int32)
    assert lib.dataflow_check(n, d, len(kind), ptr(kind), ptr(vi), ptr(vj), cols, ptr(info)) == 0
    assert lib.dataflow_check_joint(n, d, len(kind), ptr(kind), ptr(vi), ptr(vj), cols) == 0
    levels, first = int(info[0]), int(info[1])
    if cols == 0:
        assert first == levels
    if shape == "near" and n == 700:
        assert (cols < 1216) == (first > 0) or cols == 0  # narrow limits leave levels to the level form
        assert cols == 1216 or info[3] > 0 or first == levels
