"""A prepare that throws leaves no factor behind that a later one takes for its
own."""
import pytest

from conftest import rel_l2

import oracle as O
from pdgb import PdSolver, SolverParams, mesh
from pdgb import _native as N
from pdgb._native import PdgbError

pytestmark = pytest.mark.gpu

# the bound of the other solve tests: some thousand float terms in trees and
# short chains, 170 units of float rounding
TOL = 1e-5


@pytest.mark.parametrize("other_dt", [1 / 120, 1 / 30])
@pytest.mark.parametrize("device", [N.PDGB_FACTOR_HOST, N.PDGB_FACTOR_GPU])
def test_levels_after_a_refused_dsm_solve(device, other_dt):
    """Prepared, then refused with the DSM schedule (and another dt), then as at
    first: the steps are those of the first system, the levels of the first tree."""
    body = mesh.make_grid_body(18, 18, 18, young=1e5, jitter=0.1, seed=3)
    params = SolverParams(num_iterations=4, solver=1)
    with PdSolver(body, params) as e:
        e.set_factor_device(device)
        e.set_solve_mode(N.PDGB_SOLVE_LEVELS)
        e.prepare()
        first = e.factor_info()
        e.set_params(SolverParams(num_iterations=4, solver=1, dt=other_dt))
        e.set_solve_mode(N.PDGB_SOLVE_DSM)
        for _ in range(2):  # refused anew each time
            with pytest.raises(PdgbError, match="does not fit"):
                e.prepare()
        e.set_params(params)
        e.set_solve_mode(N.PDGB_SOLVE_LEVELS)
        e.update(3)
        X, _ = e.download_state()
        info = e.factor_info()
    assert (info["num_supernodes"], info["num_levels"], info["m_entries"]) == \
        (first["num_supernodes"], first["num_levels"], first["m_entries"])
    Xo, _, _ = O.simulate(body, params, 3, precision=64)
    assert rel_l2(X, Xo) < TOL
