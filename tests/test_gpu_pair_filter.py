"""The pairwise consistency test on the GPU at the sizes where the FP32 filter
takes over (65,536 pairs: 363 closures), at tile edges, with new rows only,
with a row stride of its own and with inputs that the filter must leave to the
exact test: adjacency bit for bit the oracle's."""
import numpy as np
import pytest

from oracle import rpgo_oracle as O
from rpgo_gb300 import capi
from test_pair_filter_cpu import exact, group, group2

pytestmark = pytest.mark.gpu


def _cut(g, n):
    return {k: (np.ascontiguousarray(v[:n]) if k in ("sa", "sb", "flip", "z", "zc") else v) for k, v in g.items()}


@pytest.fixture(scope="module")
def closures():
    g = group(3000, 520, 240, 3)
    rng = np.random.default_rng(4)
    n = len(g["sa"])
    assert n >= 700
    g["flip"] = (rng.random(n) < 0.2).astype(np.uint8)
    for k in rng.choice(n, 8, replace=False):
        g["zc"][k][0, 0] = np.nan
    for k in rng.choice(n, 6, replace=False):
        g["sb"][k] = g["sa"][k]
    for s in rng.choice(3000, 30, replace=False):
        g["cov"][s][1, 4] += 1e-3
    for s in rng.choice(3000, 30, replace=False):
        g["rot"][s] = 0
    return g


def _words(g, th):
    return np.asarray(O.pairwise_adjacency(3, 0, g["sa"], g["sb"], g["flip"], g["z"], g["zc"], g["pose"], g["cov"],
                                           np.zeros(len(g["rot"]), np.int32), g["rot"], th, 0.0))


@pytest.mark.parametrize("n", [362, 363, 384, 385, 408, 700])
@pytest.mark.parametrize("th", [5.0, 0.4])
def test_adjacency_is_the_oracles(closures, n, th):
    g = _cut(closures, n)
    got = capi.pairwise_adjacency(3, 0, g["sa"], g["sb"], g["flip"], g["z"], g["zc"], g["pose"], g["cov"],
                                  np.zeros(len(g["rot"]), np.int32), g["rot"], th, 0.0)
    assert np.array_equal(got, _words(g, th))


@pytest.mark.parametrize("row_begin,extra", [(0, 3), (250, 0), (333, 5), (661, 1)])
def test_new_rows_and_stride(closures, row_begin, extra):
    import torch

    n, g = 700, _cut(closures, 700)
    want = _words(g, 5.0)
    words = want.shape[1] + extra
    t = {k: torch.from_numpy(v).cuda() for k, v in g.items()}
    node = torch.zeros(len(g["rot"]), dtype=torch.int32, device="cuda")
    adj = torch.zeros(n, words, dtype=torch.int32, device="cuda")
    for first in ([0, row_begin] if row_begin else [0]):  # the group's earlier rows first, as a user has them
        rows = row_begin if first == 0 and row_begin else n
        rc = capi.load().rpgo_pairwise_adjacency_dev(
            3, 0, rows, first, t["sa"].data_ptr(), t["sb"].data_ptr(), t["flip"].data_ptr(), t["z"].data_ptr(),
            t["zc"].data_ptr(), t["pose"].data_ptr(), t["cov"].data_ptr(), node.data_ptr(), t["rot"].data_ptr(), 5.0,
            0.0, adj.data_ptr(), words, None)
        assert rc == 0
    got = adj.cpu().numpy().view(np.uint32)[:, :want.shape[1]]
    assert np.array_equal(got, want)


@pytest.mark.parametrize("n", [362, 363, 385, 700])
@pytest.mark.parametrize("th", [5.0, 0.4])
def test_adjacency_is_the_oracles_2d(n, th):
    g = group2(3000, 520, 240, 3)
    rng = np.random.default_rng(6)
    m = len(g["sa"])
    assert m >= 700
    g["flip"] = (rng.random(m) < 0.2).astype(np.uint8)
    for k in rng.choice(m, 8, replace=False):
        g["zc"][k][0, 0] = np.nan
    for k in rng.choice(m, 6, replace=False):
        g["sb"][k] = g["sa"][k]
    for s in rng.choice(3000, 30, replace=False):
        g["rot"][s] = 0
    g = _cut(g, n)
    got = capi.pairwise_adjacency(2, 0, g["sa"], g["sb"], g["flip"], g["z"], g["zc"], g["pose"], g["cov"],
                                  np.zeros(len(g["rot"]), np.int32), g["rot"], th, 0.0)
    got = np.unpackbits(np.asarray(got).view(np.uint8).reshape(n, -1), axis=1, bitorder="little")[:, :n]
    assert np.array_equal(got, exact(g, th))
