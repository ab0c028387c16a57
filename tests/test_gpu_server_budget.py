"""Cholesky requests whose tree of few levels would not fit the server's budget
get one that stores less instead of being refused."""
import time

import pytest

from conftest import rel_l2

import oracle as O
from pdgb import PdServer, SolverParams, mesh
from pdgb import _native as N

pytestmark = pytest.mark.gpu


# what a request of the mesh takes with supernodes merged only where that stores
# next to nothing more
@pytest.mark.parametrize("dims,budget", [((2, 2, 2), 12024), ((6, 6, 6), 177456), ((10, 10, 10), 897992),
                                         ((16, 16, 16), 4659180), ((60, 6, 3), 874776), ((1, 1, 300), 1517896),
                                         ((40, 3, 3), 359412)])
@pytest.mark.parametrize("cache", [0, -1])
def test_a_small_budget_takes_what_it_can_hold(dims, budget, cache):
    body = mesh.make_grid_body(*dims, young=1e5, jitter=0.1, seed=3)
    params = SolverParams(num_iterations=4, solver=1)
    with PdServer(params, hbm_budget_bytes=budget, cache_entries=cache) as srv:
        ids = [srv.submit(body, 3) for _ in range(2)]
        deadline = time.monotonic() + 60.0
        while time.monotonic() < deadline and not all(srv.poll(i)[0] in (N.PDGB_REQ_DONE, N.PDGB_REQ_FAILED)
                                                      for i in ids):
            srv.tick()
            assert srv.stats()["bytes_in_use"] <= budget
        assert [srv.poll(i) for i in ids] == [(N.PDGB_REQ_DONE, 3)] * 2
        Xo, _, _ = O.simulate(body, params, 3, precision=64)
        for i in ids:
            assert rel_l2(srv.result(i)[0], Xo) < 1e-5  # float sums of some hundred terms
