"""The collision tree's order by body and by space: the same candidates, times and
normals as the CPU query on both sides of where it changes (the bodies' boxes
together more than four times the scene's)."""
import numpy as np
import pytest

import oracle as O
from pdgb import PdSolver, SolverParams, ccd_detect, mesh, meshio

pytestmark = pytest.mark.gpu


def _soup(n, bodies, room, flat, apart, seed=3):
    rng = np.random.default_rng(seed)
    body = rng.integers(0, bodies, n).astype(np.int32)
    cent = rng.uniform(-room, room, (n, 1, 3))
    cent[:, 0, 0] += apart * body
    X = cent + rng.uniform(-0.06, 0.06, (n, 3, 3))
    if flat:
        X[..., 2] = 0.25  # one plane, and the motion leaves it
    X = X.reshape(-1, 3).astype(np.float32)
    XT = (X + rng.uniform(-0.08, 0.08, X.shape)).astype(np.float32)
    return np.arange(3 * n, dtype=np.uint32).reshape(-1, 3), body, X, XT


def _check(args):
    tI, nrm, info = ccd_detect(*args)
    tIo, nrmo, (pairs, _, marked) = O.ccd_detect(*args)
    assert info["candidate_pairs"] == pairs and info["vertices_hit"] == marked
    assert np.array_equal(tI, tIo)  # the same float operations decide both
    assert np.abs(nrm - nrmo).max() <= 1e-6


@pytest.mark.parametrize("n,bodies,room,flat,apart", [(700, 3, 0.6, False, 0.0), (700, 5, 0.6, False, 0.0),
                                                      (1500, 60, 0.8, False, 0.0), (700, 700, 0.5, False, 0.0),
                                                      (900, 6, 0.9, True, 0.0), (900, 6, 0.6, False, 0.7),
                                                      (3, 3, 0.0, False, 0.0)])
def test_mixed_and_separate_bodies(n, bodies, room, flat, apart):
    _check(_soup(n, bodies, room, flat, apart))



def test_bodies_that_leave_the_places_they_were_ordered_at():
    """150 bodies in one place when the surface is set, then scattered, then thrown:
    the tree is ordered anew on the way, and every step's candidates and times are
    the CPU query's."""
    rng = np.random.default_rng(5)
    g = mesh.make_grid_body(2, 2, 2, young=1e5, pin=None)
    n, nv = 150, g.num_verts
    t = meshio.surface_triangles(g.tets)
    tris = (t[None] + (np.arange(n) * nv)[:, None, None]).reshape(-1, 3).astype(np.uint32)
    body = np.repeat(np.arange(n, dtype=np.int32), len(t))
    X = (g.X[None] + rng.uniform(-3.0, 3.0, (n, 1, 3))).reshape(-1, 3).astype(np.float32)
    V = np.repeat(rng.normal(size=(n, 3)) * 20.0, nv, 0).astype(np.float32)
    with PdSolver([g] * n, SolverParams(num_iterations=4, solver=0)) as e:
        e.set_collision_surface(tris, body)
        e.enable_collision()
        e.upload_state(X, V)
        for _ in range(5):
            X, _ = e.download_state()
            e.update(1)
            tI, _, info = e.collision()
            tIo, _, (pairs, _, marked) = O.ccd_detect(tris, body, X, e.download_xtilde())
            assert info["candidate_pairs"] == pairs and info["vertices_hit"] == marked
            assert np.array_equal(tI, tIo)
