"""The allocation-free step's forms that a large GPU does not reach, and its bounded
wait."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_l2

import oracle as O
from pdgb import SolverParams, mesh
from pdgb import _native as N

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

PARAMS = SolverParams(num_iterations=13, rho=0.9995, solver=0)


def _call(body, dev, steps, max_ctas, missing=0, spin_limit=1 << 22):
    m = N.pdgb_noalloc_mesh(body.num_verts, body.num_tets, dev["tets"].data_ptr(), dev["X"].data_ptr(),
                            dev["mass"].data_ptr(), dev["mu"].data_ptr(), dev["dbc"].data_ptr())
    X, V = dev["X"].clone(), torch.zeros_like(dev["X"])
    st = N.lib().pdgb_noalloc_check(C.byref(m), C.byref(PARAMS.to_c()), X.data_ptr(), V.data_ptr(), steps,
                                    torch.cuda.current_stream().cuda_stream, max_ctas, missing, spin_limit)
    return st, X.cpu().numpy()


def _device(body):
    return {k: torch.from_numpy(np.ascontiguousarray(getattr(body, k))).cuda() for k in ("X", "tets", "mass", "mu", "dbc")}


# 1,024 threads a CTA walk tets and vertices in strides: one CTA, a remainder, one
# tet more than threads; and limits that leave a thread a tet
@pytest.mark.parametrize("dims,ctas", [((8, 6, 5), 1), ((11, 10, 10), 2), ((12, 9, 10), 3), ((41, 5, 5), 5),
                                       ((12, 9, 10), 6), ((12, 9, 10), 21), ((12, 9, 10), 22)])
def test_fewer_ctas_than_tets_ask_for(dims, ctas):
    body = mesh.make_grid_body(*dims, young=2e5, jitter=0.1, seed=12)
    st, X = _call(body, _device(body), 2, ctas)
    assert st == N.PDGB_OK
    Xo, _, _ = O.simulate(body, PARAMS, 2, precision=64)
    assert rel_l2(X, Xo) < 1e-5  # the bound of the other forms


@pytest.mark.parametrize("ctas", [0, 2])
def test_a_wait_that_runs_out_is_an_error_and_the_next_call_is_right(ctas):
    body = mesh.make_grid_body(12, 9, 10, young=2e5, jitter=0.1, seed=12)
    dev = _device(body)
    st, _ = _call(body, dev, 1000, ctas, missing=1, spin_limit=2000)  # one launch and the next do nothing more
    assert st == N.PDGB_ERR_TIMEOUT
    st, X = _call(body, dev, 2, ctas)
    assert st == N.PDGB_OK
    Xo, _, _ = O.simulate(body, PARAMS, 2, precision=64)
    assert rel_l2(X, Xo) < 1e-5
