"""The pairwise consistency test on the GPU on maps far from the origin of
their frame, with closures stored in both directions: adjacency bit for bit the
oracle's."""
import numpy as np
import pytest

from rpgo_gb300 import capi
from test_pair_filter_cpu import exact, group, group2
from test_pair_filter_origin_cpu import _moved

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [group, group2])
@pytest.mark.parametrize("by", [0.0, 1e5, 5e11])
def test_adjacency_far_from_the_origin(make, by):
    g = _moved(make(2500, 330, 150, 12), by)
    n, dim = len(g["sa"]), 3 if g["z"].shape[1] == 12 else 2
    assert n >= 363
    rng = np.random.default_rng(3)
    g["flip"] = (rng.random(n) < 0.3).astype(np.uint8)
    for th in (0.5, 5.0):
        got = capi.pairwise_adjacency(dim, 0, g["sa"], g["sb"], g["flip"], g["z"], g["zc"], g["pose"], g["cov"],
                                      np.zeros(len(g["rot"]), np.int32), g["rot"], th, 0.0)
        got = np.unpackbits(np.asarray(got).view(np.uint8).reshape(n, -1), axis=1, bitorder="little")[:, :n]
        assert np.array_equal(got, exact(g, th))
