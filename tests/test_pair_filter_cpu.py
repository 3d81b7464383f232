"""The FP32 pair filter (pcm_filter.cuh), run on the CPU over all pairs of a
group, against the exact verdicts of the oracle: whatever it decides must be
the exact verdict, over thresholds, directions of the closures, scales of the
noise and inputs at the edge of its premises; and on the benchmark's kind of
graph it must decide nearly everything. No GPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from oracle import rpgo_oracle as O
from rpgo_gb300 import synth
from rpgo_gb300.graph import symbol


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("pf") / "libpairfilter.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "kimera-rpgo_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "pair_filter.cpp"), "-o", out], check=True)
    return C.CDLL(out)


def group(n_poses, inliers, outliers, seed, sigma_t=0.02, sigma_r=0.005):
    """Closures over a walk's trajectory: slots, measurements, trajectory."""
    a = synth.walk3d(n_poses, inliers, outliers, seed=seed, sigma_t=sigma_t, sigma_r=sigma_r).graph.arrays()
    pose, cov = [np.array([1.0, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0])], [np.zeros((6, 6))]
    for k in range(n_poses - 1):
        R, t = a["measured"][k][:9].reshape(3, 3), a["measured"][k][9:]
        ti = -R.T @ t
        A = np.zeros((6, 6))
        A[:3, :3] = A[3:, 3:] = R.T
        A[3:, :3] = np.array([[0, -ti[2], ti[1]], [ti[2], 0, -ti[0]], [-ti[1], ti[0], 0]]) @ R.T
        S = A @ cov[-1] @ A.T + a["cov"][k]
        cov.append(np.tril(S) + np.tril(S, -1).T)
        P, T = pose[-1][:9].reshape(3, 3), pose[-1][9:]
        pose.append(np.concatenate([(P @ R).reshape(9), P @ t + T]))
    base = np.uint64(symbol("a", 0))
    lc = slice(n_poses, None)
    return {"sa": (a["key1"][lc] - base).astype(np.int32), "sb": (a["key2"][lc] - base).astype(np.int32),
            "flip": np.zeros(len(a["key1"][lc]), np.uint8), "z": np.ascontiguousarray(a["measured"][lc]),
            "zc": np.ascontiguousarray(a["cov"][lc]), "pose": np.array(pose), "cov": np.array(cov),
            "rot": np.ones(n_poses, np.uint8)}


def group2(n_poses, inliers, outliers, seed, sigma_t=0.05, sigma_th=0.01):
    """The same for a 2D grid walk."""
    a = synth.grid2d(n_poses, inliers, outliers, seed=seed, sigma_t=sigma_t, sigma_th=sigma_th).graph.arrays()
    z, zc = a["measured"][:, :4], a["cov"][:, :3, :3]
    pose, cov = [np.array([1.0, 0.0, 0.0, 0.0])], [np.zeros((3, 3))]
    for k in range(n_poses - 1):
        c, s, x, y = z[k]
        A = np.array([[c, s, s * x - c * y], [-s, c, c * x + s * y], [0, 0, 1]])
        S = A @ cov[-1] @ A.T + zc[k]
        cov.append(np.tril(S) + np.tril(S, -1).T)
        C, D, X, Y = pose[-1]
        pose.append(np.array([C * c - D * s, D * c + C * s, X + C * x - D * y, Y + D * x + C * y]))
    base = np.uint64(symbol("a", 0))
    lc = slice(n_poses, None)
    return {"sa": (a["key1"][lc] - base).astype(np.int32), "sb": (a["key2"][lc] - base).astype(np.int32),
            "flip": np.zeros(len(a["key1"][lc]), np.uint8), "z": np.ascontiguousarray(z[lc]),
            "zc": np.ascontiguousarray(zc[lc]), "pose": np.array(pose), "cov": np.array(cov),
            "rot": np.ones(n_poses, np.uint8)}


def exact(g, th):
    n = len(g["sa"])
    dim = 3 if g["z"].shape[1] == 12 else 2
    adj = np.asarray(O.pairwise_adjacency(dim, 0, g["sa"], g["sb"], g["flip"], g["z"], g["zc"], g["pose"], g["cov"],
                                          np.zeros(len(g["rot"]), np.int32), g["rot"], th, 0.0))
    return np.unpackbits(adj.view(np.uint8).reshape(n, -1), axis=1, bitorder="little")[:, :n]


def check(lib, g, th):
    """The filter's verdicts where it is sure are the exact ones; the share it leaves."""
    n = len(g["sa"])
    out = np.full((n, n), 9, np.uint8)
    p = lambda x: x.ctypes.data_as(C.c_void_p)
    lib.pair_filter(3 if g["z"].shape[1] == 12 else 2, n, p(g["sa"]), p(g["sb"]), p(g["flip"]), p(g["z"]), p(g["zc"]), p(g["pose"]), p(g["cov"]),
                    p(g["rot"]), C.c_double(th), p(out))
    low = np.tril_indices(n, -1)
    got, want = out[low], exact(g, th)[low]
    assert got.max() <= 2
    assert np.array_equal(got[got < 2], want[got < 2])
    return float(np.mean(got == 2))


@pytest.mark.parametrize("n,inliers,outliers,th", [(300, 60, 20, 5.0), (2000, 260, 90, 5.0), (2000, 260, 90, 0.3),
                                                   (2000, 260, 90, 20.0), (12000, 300, 150, 5.0)])
def test_decides_nearly_every_pair(lib, n, inliers, outliers, th):
    assert check(lib, group(n, inliers, outliers, n), th) < 0.05


@pytest.mark.parametrize("sigma_t,sigma_r", [(2e-5, 5e-6), (2.0, 0.3), (0.02, 1e-9), (1e-10, 0.005), (1e-12, 1e-12),
                                             (3e3, 0.005)])
def test_scales_of_the_noise(lib, sigma_t, sigma_r):
    g = group(700, 140, 60, 5, sigma_t, sigma_r)
    for th in (0.1, 3.0):
        check(lib, g, th)


def test_directions(lib):
    g = group(900, 180, 80, 6)
    g["flip"] = (np.random.default_rng(2).random(len(g["sa"])) < 0.5).astype(np.uint8)
    assert check(lib, g, 5.0) < 0.05


def test_inputs_at_the_edge_of_the_premises(lib):
    rng = np.random.default_rng(9)
    g = group(800, 150, 50, 8)
    n = len(g["sa"])
    pick = lambda k: rng.choice(n, k, replace=False)
    for k in pick(6):  # the same endpoints as another closure, and one pose twice
        g["sa"][k], g["sb"][k] = g["sa"][(k + 1) % n], g["sb"][(k + 1) % n]
    for k in pick(4):
        g["sb"][k] = g["sa"][k]
    for k in pick(8):  # rotations by nearly and exactly pi
        w = rng.normal(size=3)
        w *= (np.pi - rng.choice([0.0, 1e-9, 1e-6, 1e-4, 1e-2])) / np.linalg.norm(w)
        g["z"][k][:9] = synth.so3_exp(w).reshape(9)
    for k in pick(3):
        g["zc"][k] = 0.0
    for k in pick(3):
        g["zc"][k][0, 0] = np.nan  # rotation information missing
    for k in pick(3):
        g["zc"][k] *= 1e30
    for k in pick(2):
        g["z"][k][9:] = 1e20
    for k in pick(2):
        g["z"][k][:9] *= 1.0 + 1e-4  # not quite a rotation
    for s in rng.choice(800, 6, replace=False):  # trajectory covariances
        g["cov"][s][2, 5] += 1e-3
    for s in rng.choice(800, 4, replace=False):
        g["cov"][s] = -g["cov"][s]
    for s in rng.choice(800, 4, replace=False):
        g["rot"][s] = 0
    for th in (0.5, 5.0):
        check(lib, g, th)


@pytest.mark.parametrize("n,inliers,outliers,th", [(300, 60, 20, 5.0), (2000, 260, 90, 5.0), (2000, 260, 90, 0.3),
                                                   (2000, 260, 90, 20.0), (6000, 300, 150, 5.0)])
def test_decides_nearly_every_pair_2d(lib, n, inliers, outliers, th):
    assert check(lib, group2(n, inliers, outliers, n), th) < 0.05


@pytest.mark.parametrize("sigma_t,sigma_r", [(2e-5, 5e-6), (2.0, 0.3), (0.02, 1e-9), (1e-10, 0.005), (1e-12, 1e-12),
                                             (3e3, 0.005)])
def test_scales_of_the_noise_2d(lib, sigma_t, sigma_r):
    g = group2(700, 140, 60, 5, sigma_t, sigma_r)
    for th in (0.1, 3.0):
        check(lib, g, th)


def test_directions_and_edges_2d(lib):
    rng = np.random.default_rng(19)
    g = group2(800, 180, 80, 8)
    n = len(g["sa"])
    g["flip"] = (rng.random(n) < 0.5).astype(np.uint8)
    assert check(lib, g, 5.0) < 0.05
    pick = lambda k: rng.choice(n, k, replace=False)
    for k in pick(6):  # the same endpoints as another closure, and one pose twice
        g["sa"][k], g["sb"][k] = g["sa"][(k + 1) % n], g["sb"][(k + 1) % n]
    for k in pick(4):
        g["sb"][k] = g["sa"][k]
    for k in pick(8):  # rotations by nearly and exactly pi
        w = np.pi - rng.choice([0.0, 1e-9, 1e-6, 1e-4, 1e-2])
        g["z"][k][:2] = np.cos(w), np.sin(w)
    for k in pick(8):  # exact repeats: loops by nearly no angle
        m = (k + 5) % n
        for v in ("sa", "sb", "flip"):
            g[v][k] = g[v][m]
        w = rng.choice([0.0, 1e-11, 1e-9, 1e-7, 1e-5])
        c, s = g["z"][m][:2]
        g["z"][k] = g["z"][m]
        g["z"][k][:2] = c * np.cos(w) - s * np.sin(w), s * np.cos(w) + c * np.sin(w)
    for k in pick(3):
        g["zc"][k] = 0.0
    for k in pick(3):
        g["zc"][k][0, 0] = np.nan  # rotation information missing
    for k in pick(3):
        g["zc"][k][2, 2] = np.nan
    for k in pick(3):
        g["zc"][k] *= 1e30
    for k in pick(2):
        g["z"][k][2:] = 1e20
    for k in pick(4):
        g["z"][k][:2] *= 1.0 + rng.choice([1e-4, 2e-8])  # not quite a rotation
    for s in rng.choice(800, 6, replace=False):  # trajectory covariances
        g["cov"][s][1, 2] += 1e-3
    for s in rng.choice(800, 4, replace=False):
        g["cov"][s] = -g["cov"][s]
    for s in rng.choice(800, 4, replace=False):
        g["rot"][s] = 0
    for th in (0.5, 5.0):
        check(lib, g, th)
