"""The layout's Morton orders (no GPU): radix-sorted, equal keys in caller
order, for sizes on both sides of its comparison-sort and threading limits; and
the system matrix the marker-array assembly builds."""
import numpy as np
import pytest

from test_capi_host import inspect
from test_cholesky_host import factor_check

import oracle as O
from pdgb import mesh
from pdgb import _native as N


def _spread(x):
    x = x.astype(np.uint64) & np.uint64(0x1FFFFF)
    for s, m in ((32, 0x1F00000000FFFF), (16, 0x1F0000FF0000FF), (8, 0x100F00F00F00F00F), (4, 0x10C30C30C30C30C3),
                 (2, 0x1249249249249249)):
        x = (x | (x << np.uint64(s))) & np.uint64(m)
    return x


def _keys(P, X):
    lo, hi = X.astype(np.float64).min(0), X.astype(np.float64).max(0)
    ext = float((hi - lo).max()) or 1.0
    q = np.clip((P - lo) * (2097151.0 / ext), 0.0, 2097151.0).astype(np.uint64)
    return _spread(q[:, 0]) | (_spread(q[:, 1]) << np.uint64(1)) | (_spread(q[:, 2]) << np.uint64(2))


# 1 tet-cell (comparison sort), around 512 keys, and past 2 x 16,384 tets (threads)
@pytest.mark.parametrize("dims,jitter", [((1, 1, 1), 0.0), ((7, 7, 7), 0.1), ((5, 4, 5), 0.1), ((6, 4, 5), 0.0),
                                         ((19, 18, 20), 0.1), ((3, 60, 41), 0.0)])
def test_orders_are_stable_morton_orders(dims, jitter):
    body = mesh.make_grid_body(*dims, jitter=jitter, seed=3)
    st, _, vperm, tperm = inspect(body)
    assert st == N.PDGB_OK
    x = body.X.astype(np.float64)
    assert np.array_equal(vperm, np.argsort(_keys(x, body.X), kind="stable"))
    c = np.zeros((body.num_tets, 3))
    for k in range(4):
        c += 0.25 * x[body.tets[:, k]]
    assert np.array_equal(tperm, np.argsort(_keys(c, body.X), kind="stable"))


def test_the_first_bad_tet_is_reported_across_threads():
    body = mesh.make_grid_body(20, 20, 20)
    body.tets = body.tets.copy()
    st, _, _, tperm = inspect(body)
    assert st == N.PDGB_OK
    for t in tperm[[9000, 39000]]:  # flat: two corners the same
        body.tets[t, 3] = body.tets[t, 2]
    st, *_ = inspect(body)
    assert st == N.PDGB_ERR_BAD_MESH
    assert b"zero rest volume" in N.lib().pdgb_last_error()


# one band (the whole tree one supernode), two and more levels; long and flat
@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 2, 2), (5, 5, 5), (11, 3, 9), (23, 2, 1), (12, 12, 12)])
def test_amalgamated_factor_solves(dims):
    body = mesh.make_grid_body(*dims, young=2e5, jitter=0.15, seed=5)
    b = np.random.default_rng(1).normal(size=(body.num_verts, 3))
    st, info, x = factor_check(body, N.PDGB_ORDER_AMD, b)
    assert st == N.PDGB_OK
    xo = O.solve3(body, 1 / 120, b)
    # blocks M_s rounded to float: 6e-8 an entry, sums of up to n of them
    assert np.linalg.norm(x - xo) < 1e-6 * np.linalg.norm(xo)
    assert 1 <= info.num_levels <= 4
