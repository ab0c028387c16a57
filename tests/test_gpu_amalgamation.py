"""The trees that a batch's bodies are amalgamated to."""
import pytest

from conftest import rel_l2

import oracle as O
from pdgb import PdSolver, SolverParams, mesh
from pdgb import _native as N

pytestmark = pytest.mark.gpu


def _per_body(n, body):
    with PdSolver([body] * n, SolverParams(num_iterations=1, solver=1)) as e:
        e.prepare()
        f = e.factor_info()
    return f["num_supernodes"] / n, f["num_levels"]


@pytest.mark.parametrize("dims", [(3, 3, 3), (6, 6, 6)])
def test_many_bodies_are_priced_like_fewer(dims):
    """A body's share of a level falls as 1 / bodies: past some thousand of them
    it is below what any item costs, and the tree stays the same from there on."""
    body = mesh.make_grid_body(*dims, young=1e5, jitter=0.1, seed=3)
    assert _per_body(3700, body) == _per_body(3900, body)


def test_the_cta_schedule_has_a_tree_of_its_own():
    """A barrier of one CTA is no launch: fewer explicit zeros and more levels than
    the per-level launches' tree -- and each schedule's steps are right when they
    are changed on the way."""
    body = mesh.make_grid_body(13, 12, 14, young=1e5, jitter=0.1, seed=3)
    params = SolverParams(num_iterations=5, solver=1)
    order = (N.PDGB_SOLVE_LEVELS, N.PDGB_SOLVE_CTA, N.PDGB_SOLVE_PERSISTENT, N.PDGB_SOLVE_CTA, N.PDGB_SOLVE_CLUSTER)
    with PdSolver(body, params) as e:
        entries = []
        for m in order:
            e.set_solve_mode(m)
            e.update(1)
            entries.append(e.factor_info()["m_entries"])
        X, _ = e.download_state()
    assert entries[0] == entries[2] == entries[4] and entries[1] == entries[3] < 0.7 * entries[0]
    Xo, _, _ = O.simulate(body, params, len(order), precision=64)
    # some thousand float terms in trees and short chains: 170 units of rounding
    assert rel_l2(X, Xo) < 1e-5
