"""One damped step of the direct solve (tests/native/solve_step.cpp): the
dataflow part gives the bits of the level form on the same CTAs, whatever its
width and the run (a level of more than 7 columns per CTA adds its backward
sums in another order than a narrower one, so the number of CTAs can change the
rounding of either form); and a wait of it that runs out ends the solve with
its status, after which the same buffers solve again."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from test_gpu_dataflow_solve import _graph

CSRC = os.path.join(ROOT, "kimera-rpgo_gb300", "csrc")
LIBDIR = os.path.join(ROOT, "kimera-rpgo_gb300", "rpgo_gb300")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from rpgo_gb300 import build

    build()
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = str(tmp_path_factory.mktemp("step") / "libsolvestep.so")
    subprocess.run([nvcc, "-O1", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-x", "c++", "-I", CSRC,
                    os.path.join(ROOT, "tests", "native", "solve_step.cpp"), "-L", LIBDIR, "-lrpgo_gb300", "-Xlinker",
                    "-rpath," + LIBDIR, "-o", out], check=True)
    return C.CDLL(out)


def _steps(lib, g, runs, joint, lam=1e-5):
    """The step, model change and status of each run (coop_ctas, df_cols, df_polls)."""
    a = g.arrays()
    dim, n = g.dim, len(a["value_keys"])
    at = {int(k): i for i, k in enumerate(a["value_keys"])}
    kind = np.ascontiguousarray(a["kind"], np.int32)
    vi = np.array([at[int(k)] for k in a["key1"]], np.int32)
    vj = np.array([at[int(k)] if c == 0 else v for k, c, v in zip(a["key2"], kind, vi)], np.int32)
    z, R, x = (np.array(a[k], np.float64) for k in ("measured", "sqrt_info", "value_poses"))
    # off the odometry, which solves a graph without closures
    x[:, -dim:] += 0.1 * np.random.default_rng(n).normal(size=(n, dim))
    m = len(runs)
    coop, cols, polls = (np.array([r[k] for r in runs], np.int32) for k in range(3))
    step = np.full((m, (2 if joint else 1) * n * g.d), np.nan)
    change, status, info = np.zeros(m), np.full(m, -1, np.int32), np.zeros(4, np.int32)
    p = lambda v: v.ctypes.data_as(C.c_void_p)
    rc = lib.solve_steps(dim, n, len(kind), p(kind), p(vi), p(vj), p(z), p(R), p(x), C.c_double(lam), int(joint), m,
                         p(coop), p(cols), p(polls), p(step), p(change), p(status), p(info))
    assert rc == 0
    return step, change, status, info


SHAPES = [(2, 0, 0), (4, 0, 0), (5, 0, 0), (9, 0, 0), (10, 3, 0), (33, 8, 0), (50, 0, 0), (130, 40, 0), (60, 0, 60),
          (400, 100, 45), (700, 150, 0)]


def test_harness_builds(lib):
    assert lib.solve_steps


@pytest.mark.gpu
@pytest.mark.parametrize("joint", [False, True])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n,closures,hub", SHAPES)
def test_same_bits_as_the_level_form(lib, dim, n, closures, hub, joint):
    g = _graph(dim, n, closures, hub, seed=n)
    runs = [(c, w, 0) for c in (0, 1, 3) for w in (0, 1, 7, -1)]
    runs += [(0, -1, 0)] * 4
    step, change, status, _ = _steps(lib, g, runs, joint)
    assert not status.any()
    assert np.isfinite(step).all() and np.abs(step).max() > 0
    for k, r in enumerate(runs):
        level = next(i for i, q in enumerate(runs) if q[0] == r[0])
        assert runs[level][1] == 0 and np.array_equal(step[k], step[level]), r
    # the model change is a sum over the CTAs: same CTAs, same bits
    assert len({change[k] for k, r in enumerate(runs) if r[0] == 0}) == 1
    if joint:
        assert np.array_equal(step[0][: len(step[0]) // 2], step[0][len(step[0]) // 2:])


@pytest.mark.gpu
@pytest.mark.parametrize("joint", [False, True])
@pytest.mark.parametrize("dim", [2, 3])
def test_a_wait_that_runs_out_is_reported(lib, dim, joint):
    g = _graph(dim, 700, 150, 0, seed=700)
    runs = [(0, -1, 0), (0, -1, 1), (0, -1, 0), (0, -1, 1), (0, -1, 0)]
    step, change, status, info = _steps(lib, g, runs, joint)
    assert info[3] < info[0]  # there is a dataflow part
    assert status.tolist() == [0, 2, 0, 2, 0]
    for k in (2, 4):
        assert np.array_equal(step[k], step[0]) and change[k] == change[0]
