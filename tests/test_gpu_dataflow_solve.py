"""The direct solve's dataflow part on the GPU at the sizes where it can go
wrong: tail only, one column, chains, a hub past the part's limits (level form
at the top), both block sizes, and one, two or three CTAs for all columns,
against the oracle's LM. Both solve the same FP64 systems and stop at the same
iterate, so poses agree to 1e-6 relative, the bound of the other parity tests
(rounding of about 1e-12 per step, amplified by the weakly held poses)."""
import numpy as np
import pytest

from oracle import rpgo_oracle as O
from rpgo_gb300 import capi, synth
from rpgo_gb300.graph import diagonal_sigmas, symbol
from rpgo_gb300.params import QUIET, RobustSolverParams

pytestmark = pytest.mark.gpu


TAIL4 = [(38, 49), (28, 39), (33, 27)]


def _graph(dim, n, closures, hub, seed):
    make = synth.walk3d if dim == 3 else synth.grid2d
    s = make(n, closures, 0, seed=seed)
    sig = np.array([0.005] * 3 + [0.02] * 3) if dim == 3 else np.array([0.05, 0.05, 0.01])
    mat = synth._T if dim == 3 else synth._M2
    vec = synth._p if dim == 3 else synth._p2
    for i, j in TAIL4 if n == 50 else []:  # a dense tail of four blocks, more entries than threads
        z = np.linalg.inv(mat(s.gt[i])) @ mat(s.gt[j])
        s.graph.add_between(symbol("a", i), symbol("a", j), vec(z), diagonal_sigmas(sig))
    for k in range(2, hub):
        z = np.linalg.inv(mat(s.gt[0])) @ mat(s.gt[k])
        s.graph.add_between(symbol("a", 0), symbol("a", k), vec(z), diagonal_sigmas(sig))
    return s.graph


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n,closures,hub", [(2, 0, 0), (4, 0, 0), (5, 0, 0), (9, 0, 0), (10, 3, 0), (33, 8, 0), (50, 0, 0),
                                            (130, 40, 0), (60, 0, 60), (400, 100, 45)])
def test_dataflow_solve_matches_the_oracle(dim, n, closures, hub):
    g = _graph(dim, n, closures, hub, seed=n)
    p = RobustSolverParams().setNoRejection(QUIET, dim)
    o = O.OracleSolver(p)
    assert o.update(g) == 0
    ko, po = o.estimate()
    s = capi.RobustSolver(p)
    assert s.update(g) == 0
    kg, pg = s.estimate()
    runs = [pg]
    for ctas in (1, 2, 3):
        status, kb, pb, _, _ = capi.solve_batch(p, [g], workers=1, coop_ctas=ctas)[0]
        assert status == 0 and np.array_equal(kb, ko)
        runs.append(pb)
    assert np.array_equal(kg, ko)
    for x in runs:
        assert np.max(np.abs(x - po) / np.maximum(1.0, np.abs(po))) <= 1e-6
    # the step of every damped system is the level form's whatever the width
    # of the dataflow part, so the number of CTAs changes rounding at most
    for x in runs[1:]:
        assert np.max(np.abs(x - pg) / np.maximum(1.0, np.abs(pg))) <= 1e-9
