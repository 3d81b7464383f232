"""The FP32 pair filter where the map is far from the origin of its frame: its
verdicts stay the exact ones, and it decides as many pairs as beside the
origin; with two robots whose frames are far apart, closures stored in both
directions, steps of a kilometre, and noise so small that the rounding of the
positions is what the bounds have to cover. No GPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from test_pair_filter_cpu import check, group, group2


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("pf") / "libpairfilterorigin.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "kimera-rpgo_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "pair_filter_origin.cpp"), "-o", out], check=True)
    return C.CDLL(out)


def _moved(g, by, slots=slice(None)):
    """The trajectory (those slots of it) moved in its frame."""
    dim = 3 if g["z"].shape[1] == 12 else 2
    g["pose"][slots, 9 if dim == 3 else 2:] += np.asarray([1.0, -0.6, 0.3][:dim]) * by
    return g


def _turned(g, slots, angle):
    """Those slots' frame turned about z (rotation and translation)."""
    c, s = np.cos(angle), np.sin(angle)
    Z = np.array([[c, -s, 0], [s, c, 0], [0, 0, 1]])
    for k in slots:
        p = g["pose"][k]
        if len(p) == 12:
            p[:9], p[9:] = (Z @ p[:9].reshape(3, 3)).reshape(9), Z @ p[9:]
        else:
            p[:] = c * p[0] - s * p[1], s * p[0] + c * p[1], c * p[2] - s * p[3], s * p[2] + c * p[3]
    return g


@pytest.mark.parametrize("make,th", [(group, 5.0), (group2, 1.0)])
@pytest.mark.parametrize("by", [0.0, 1e3, 1e5, 5e6])
def test_share_does_not_grow_with_the_distance(lib, make, th, by):
    assert check(lib, _moved(make(2000, 260, 90, 2000), by), th) < 0.05


@pytest.mark.parametrize("make", [group, group2])
def test_two_frames_and_directions(lib, make):
    g = make(900, 180, 80, 6)
    n, m = len(g["sa"]), len(g["rot"])
    for v in ("pose", "cov", "rot"):  # the second robot: the same walk in a frame of its own
        g[v] = np.concatenate([g[v], g[v]])
    g["sb"] = g["sb"] + np.int32(m)
    _turned(_moved(g, 3e5, slice(m, None)), range(m, 2 * m), 0.7)
    _moved(g, -4e6, slice(0, m))
    g["flip"] = (np.random.default_rng(2).random(n) < 0.4).astype(np.uint8)
    back = g["flip"] == 1
    g["sa"][back], g["sb"][back] = g["sb"][back], g["sa"][back]  # stored from robot b to robot a
    for k in np.nonzero(back)[0]:  # the measurement's inverse
        z = g["z"][k]
        if len(z) == 12:
            R, t = z[:9].reshape(3, 3).copy(), z[9:].copy()
            z[:9], z[9:] = R.T.reshape(9), -R.T @ t
        else:
            c, s, x, y = z
            z[:] = c, -s, -c * x - s * y, s * x - c * y
    for th in (0.5, 5.0):
        assert check(lib, g, th) < 0.05


@pytest.mark.parametrize("make", [group, group2])
@pytest.mark.parametrize("sigma_t,sigma_r", [(1e-9, 0.2), (1e-12, 1e-12), (1e-7, 1e-9), (0.02, 1e-9), (50.0, 0.3)])
@pytest.mark.parametrize("by", [0.0, 1e8, 5e11])
def test_verdicts_at_the_limits_of_the_rounding(lib, make, sigma_t, sigma_r, by):
    g = _moved(make(500, 110, 50, 5, sigma_t, sigma_r), by)
    g["pose"][250:, -2] += 1e3 * by ** 0.5  # and far from closure 0
    for th in (0.1, 3.0):
        check(lib, g, th)


@pytest.mark.parametrize("make", [group, group2])
def test_without_a_finite_origin(lib, make):
    g = make(400, 90, 30, 7)
    g["pose"][g["sa"][0], -1] = np.inf
    g["pose"][g["sb"][0], -2] = np.nan
    assert check(lib, g, 5.0) < 0.1
    g = make(400, 90, 30, 7)
    g["pose"][g["sb"][0], -1] = 1e300
    assert check(lib, g, 5.0) < 0.1


def test_no_verdict_on_a_covariance_that_may_be_indefinite(lib):
    """Far beyond the threshold, with a relative error of the covariance (here
    1.1 * 64 * 2^-24 * ph^2) on both sides of 1."""
    f = [C.c_float(x) for x in (100.0, 100.0, 100.0, 0.0, 0.0)]
    rest = [C.c_float(x) for x in (0.0, 0.0, 1.0)]
    assert lib.pair_decide(*f, C.c_float(480.0), *rest) == 0  # 0.97
    assert lib.pair_decide(*f, C.c_float(500.0), *rest) == 2  # 1.05
    assert lib.pair_decide(*f, C.c_float(float("nan")), *rest) == 2


@pytest.mark.parametrize("make", [group, group2])
def test_indefinite_closure_covariances(lib, make):
    g = make(700, 140, 60, 11)
    d = g["zc"].shape[1]
    for k in range(0, len(g["sa"]), 2):
        s = np.sqrt(np.diag(g["zc"][k])) * 10.0 ** (k % 5)
        g["zc"][k] = np.outer(s, s) * (-0.95 + 0.05 * (k % 3))
        g["zc"][k][np.diag_indices(d)] = s * s
    for th in (0.01, 0.5, 5.0, 100.0):
        check(lib, g, th)
