"""The elimination order at the size where it stops counting in the tree's
level (12,288 unknowns): on both sides every column structure and task list
holds, and up to it a long trajectory with local closures has a tree no deeper
than two levels per doubling of its length. No GPU."""
import ctypes as C

import numpy as np
import pytest

from test_plan_symbolic_cpu import _edges, _p, _pose_graph, lib  # noqa: F401


@pytest.mark.parametrize("d,n", [(6, 2), (6, 300), (6, 2048), (6, 2049), (3, 500), (3, 4096), (3, 4097)])
def test_tree_depth(lib, d, n):  # noqa: F811
    rng = np.random.default_rng(n)
    ei, ej = _edges(_pose_graph(n, n // 6, 30, rng))
    levels = C.c_int(0)
    assert lib.plan_task_order_check(n, d, len(ei), _p(ei), _p(ej), C.byref(levels)) == 0
    if n * d <= 12288:
        assert levels.value <= 2 * np.ceil(np.log2(n)) + 1
