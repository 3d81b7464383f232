"""The FP32 log map of the pair filter (pcm_filter.cuh) against the exact
test's formulas in 64 bits: wherever it calls itself certain, each entry is
within its bound. The formulas change at an angle (cos = -0.8) and, near pi,
with the largest diagonal entry; for a matrix that is not quite a rotation (a
chain of rounded rotations, say) the two sides of such a line differ. No GPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("pl") / "libpairlogmap.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "kimera-rpgo_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "pair_filter_logmap.cpp"), "-o", out], check=True)
    return C.CDLL(out)


def log_exact(R, t):
    """p3_logmap of pcm_math.cuh (n poses)."""
    v = np.stack([R[:, 2, 1] - R[:, 1, 2], R[:, 0, 2] - R[:, 2, 0], R[:, 1, 0] - R[:, 0, 1]], 1)
    cs, sn = np.trace(R, axis1=1, axis2=2) - 1.0, np.linalg.norm(v, axis=1)
    th = np.arctan2(sn, cs)
    s, c, omc = 0.5 * sn, 0.5 * cs, 1.0 - 0.5 * cs
    t2 = th * th
    with np.errstate(all="ignore"):
        w = v * np.where(th < 0.01, (7 / 720 * t2 + 1 / 12) * t2 + 0.5, th / sn)[:, None]
        d = np.stack([R[:, 0, 0], R[:, 1, 1], R[:, 2, 2]], 1)
        i = np.where(d[:, 1] > d[:, 0], 1, 0)
        k = np.arange(len(R))
        i = np.where(d[:, 2] > d[k, i], 2, i)
        ni = np.sqrt((d[k, i] - c) / omc)
        n = (R[k, i] + R[k, :, i]) / (2.0 * omc * ni)[:, None]
        n[k, i] = ni
        f = np.where(np.sum(n * v, 1) < 0.0, -th, th)
        w = np.where((cs > -1.6)[:, None], w, f[:, None] * n)
        beta = np.where(th < 0.01, (t2 / 30240 + 1 / 720) * t2 + 1 / 12, (1.0 - th * s / (s * s + omc * omc)) / t2)
    W = np.cross(w, t)
    return np.concatenate([w, t - 0.5 * W + beta[:, None] * np.cross(w, W)], 1)


def poses(n, seed, shear, whole):
    """Rotations over all angles, many of them where the formulas change, off
    by `shear` in their symmetric part (which the filter's check of the
    rotation does not see) and by `whole` in every entry."""
    g = np.random.default_rng(seed)
    a = g.normal(size=(n, 3))
    k = np.arange(n)
    a[k % 5 == 0, 1] = a[k % 5 == 0, 0]  # equal diagonal entries
    a[k % 7 == 0, 2] = -a[k % 7 == 0, 1]
    a[k % 3 == 0, 0] *= 1e-3
    a /= np.linalg.norm(a, axis=1)[:, None]
    u = g.uniform(-1, 1, n)
    th = np.choose(k % 5, [np.pi * (u + 1) / 2, 10 ** (-8 + 4 * (u + 1)), np.pi - 10 ** (-7 + 3 * (u + 1)),
                           np.arccos(-0.8) + 1e-6 * u, 0.01 + 1e-5 * u])
    K = np.zeros((n, 3, 3))
    K[:, 0, 1], K[:, 0, 2], K[:, 1, 2] = -a[:, 2], a[:, 1], -a[:, 0]
    K -= K.transpose(0, 2, 1)
    R = (np.cos(th)[:, None, None] * np.eye(3) + (1 - np.cos(th))[:, None, None] * a[:, :, None] * a[:, None, :]
         + np.sin(th)[:, None, None] * K)
    E = g.uniform(-shear, shear, (n, 3, 3))
    E = np.tril(E, -1)
    return R + E + E.transpose(0, 2, 1) + g.uniform(-whole, whole, (n, 3, 3)), g.normal(size=(n, 3)) * 10 ** g.uniform(
        -3, 3, (n, 1))


@pytest.mark.parametrize("shear,whole", [(0.0, 0.0), (1e-6, 0.0), (1e-5, 0.0), (1e-3, 0.0), (0.0, 1e-6), (0.0, 3e-6)])
def test_certain_log_maps_are_within_their_bounds(lib, shear, whole):
    n = 400_000
    R, t = poses(n, 3, shear, whole)
    pose = np.ascontiguousarray(np.concatenate([R.reshape(n, 9), t], 1))
    xi, e, ok = np.zeros((n, 6), np.float32), np.zeros((n, 2), np.float32), np.zeros(n, np.uint8)
    p = lambda x: x.ctypes.data_as(C.c_void_p)
    lib.pair_logmap(n, p(pose), p(xi), p(e), p(ok))
    err, sure = np.abs(xi - log_exact(R, t)), ok == 1
    assert sure.mean() > 0.2
    assert np.all(err[sure, :3] <= e[sure, :1]) and np.all(err[sure, 3:] <= e[sure, 1:])
