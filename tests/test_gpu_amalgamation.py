"""The trees that a batch's bodies are amalgamated to."""
import pytest

from pdgb import PdSolver, SolverParams, mesh

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
