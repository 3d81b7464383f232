"""The trajectory scan on the device against the oracle's composition, entry
by entry (bit for bit): lengths around its chunk of 16 steps, chains that
continue from older poses, two robots step about, a slot written twice, a
start covariance that is not symmetric, missing rotation information."""
import numpy as np
import pytest

from oracle import rpgo_oracle as O
from rpgo_gb300 import capi, synth

pytestmark = pytest.mark.gpu


def _slots(kind, n):
    if kind == "chain":
        return np.arange(n), np.arange(1, n + 1)
    if kind == "branches":  # every few steps from an older pose
        src = np.arange(n)
        for k in range(3, n, 5):
            src[k] = (k * 7) % k
        return src, np.arange(1, n + 1)
    if kind == "robots":  # two chains in turn, from slots 0 and 1
        src = np.arange(n)
        return src, src + 2
    src, dst = np.arange(n), np.arange(1, n + 1)  # slots written twice
    for k in range(4, n, 6):
        dst[k] = max(1, k - 2)
        if k + 1 < n:
            src[k + 1] = dst[k]
    return src, dst


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("kind,n", [("chain", 1), ("chain", 15), ("chain", 16), ("chain", 17), ("chain", 65),
                                    ("branches", 33), ("branches", 80), ("robots", 50), ("twice", 49)])
def test_scan_is_the_oracles_composition(dim, mode, kind, n):
    import torch

    rng = np.random.default_rng(100 * n + dim)
    st, d = (12, 6) if dim == 3 else (4, 3)
    if dim == 3:
        dp = np.array([np.concatenate([synth.so3_exp(rng.normal(0, 0.4, 3)).reshape(9), rng.normal(0, 2, 3)])
                       for _ in range(n)])
    else:
        th = rng.normal(0, 0.5, n)
        dp = np.stack([np.cos(th), np.sin(th), rng.normal(0, 2, n), rng.normal(0, 2, n)], axis=1)
    A = rng.normal(0, 0.1, (n, d, d))
    dc = A @ A.transpose(0, 2, 1) + 1e-4 * np.eye(d)
    if n > 20:
        dc[n // 2][0, 0] = np.nan  # no rotation information (2D: the first entry as well)
    src, dst = (x.astype(np.int32) for x in _slots(kind, n))
    slots = int(max(src.max(), dst.max())) + 1
    pose, cov = np.zeros((slots, st)), np.zeros((slots, d, d))
    pose[:, [0, 4, 8] if dim == 3 else [0]] = 1.0
    cov[0] = rng.normal(0, 0.1, (d, d))  # what a caller's slot may hold: not symmetric
    node, rot = np.zeros(slots, np.int32), np.ones(slots, np.uint8)
    t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    D = [t(x) for x in (src, dst, dp, dc, pose, cov, node, rot)]
    assert capi.load().rpgo_trajectory_scan_dev(dim, mode, n, *[x.data_ptr() for x in D], None) == 0
    got_pose, got_cov, got_node, got_rot = (x.cpu().numpy() for x in D[4:])
    rd = 3 if dim == 3 else 1
    for k in range(n):
        zc, zr = dc[k].copy(), 1
        if np.isnan(zc[0, 0]):
            zr = 0
            zc[:rd, :] = 0.0
            zc[:, :rd] = 0.0
        p, c, r = O.pwc_op(dim, 0, pose[src[k]], cov[src[k]], int(rot[src[k]]), dp[k], zc, zr)
        pose[dst[k]], cov[dst[k]], rot[dst[k]], node[dst[k]] = p, c, r, node[src[k]] + 1
    assert np.array_equal(got_pose, pose)
    assert np.array_equal(got_rot, rot)
    if mode == 0:
        assert np.array_equal(got_cov, cov)
    else:
        assert np.array_equal(got_node, node)
