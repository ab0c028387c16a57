"""Which bad tet the layout reports where several threads find one each (no GPU):
the first in its own order, as one loop would."""
import numpy as np
import pytest

from test_capi_host import inspect
from test_layout_order import _keys

from pdgb import mesh
from pdgb import _native as N

FLAT, WEIGHT = b"zero rest volume", b"negative or non-finite weight"


def _order(body):
    c = np.zeros((body.num_tets, 3))
    for k in range(4):
        c += 0.25 * body.X.astype(np.float64)[body.tets[:, k]]
    return np.argsort(_keys(c, body.X), kind="stable")


# 40,000 tets are two parts, 80,000 four; first and last part, neighbours, one part
@pytest.mark.parametrize("n,at", [(20, (300, 39700)), (20, (19990, 20010)), (20, (9000, 9001)), (25, (100, 77000)),
                                  (25, (25000, 45000))])
@pytest.mark.parametrize("kinds", [(FLAT, WEIGHT), (WEIGHT, FLAT), (FLAT, FLAT), (WEIGHT, WEIGHT)])
def test_the_first_in_the_layouts_order_is_named(n, at, kinds):
    body = mesh.make_grid_body(n, n, n, jitter=0.1, seed=2)
    body.tets, body.mu = body.tets.copy(), body.mu.copy()
    bad = _order(body)[list(at)]
    for t, kind in zip(bad, kinds):
        if kind is FLAT:
            body.tets[t, 3] = body.tets[t, 2]  # moves the tet a little along the curve
        else:
            body.mu[t] = -1.0
    place = {int(t): p for p, t in enumerate(_order(body))}
    first = min(range(2), key=lambda i: place[int(bad[i])])
    st, *_ = inspect(body)
    assert st == N.PDGB_ERR_BAD_MESH
    msg = N.lib().pdgb_last_error()
    assert b"tet %d " % bad[first] in msg and kinds[first] in msg, msg
