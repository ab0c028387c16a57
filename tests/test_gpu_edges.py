"""Kernels at the sizes where their splits change: tiles and warps of the
triangular solves, panels of the factorisation, the allocation-free step's
launch shapes, the iterate buffers that take turns, the collision query's
thresholds -- each against the FP64 oracle, the host factor or the CPU query."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_l2

import oracle as O
from pdgb import PdSolver, SolverParams, ccd_detect, mesh
from pdgb import _native as N

pytestmark = pytest.mark.gpu

# Positions are a few metres at most and every sum of a solve has at most some
# thousand float terms in trees and short chains: 1e-5 relative is 170 units
# of float rounding.
TOL = 1e-5


def _against_oracle(e, body, params, steps):
    e.update(steps)
    X, _ = e.download_state()
    Xo, _, _ = O.simulate(body, params, steps, precision=64)
    assert rel_l2(X, Xo) < TOL, rel_l2(X, Xo)


# One dense supernode of n vertices: n = 8 .. 63 a warp or one tile, 64 the
# least tile, 128 / 130 one and two row tiles, 96 / 100 three and four column
# tiles, 256 / 260 two and three rows of tiles.
@pytest.mark.parametrize("dims", [(1, 1, 1), (1, 1, 6), (1, 1, 7), (2, 2, 2), (2, 2, 6), (3, 3, 3), (1, 5, 7), (1, 4, 9),
                                  (1, 7, 7), (1, 4, 12), (3, 7, 7), (1, 9, 12)])
def test_dense_solve_at_tile_edges(dims):
    body = mesh.make_grid_body(*dims, young=1e5, jitter=0.1, seed=7)
    params = SolverParams(num_iterations=6, solver=1)
    with PdSolver(body, params) as e:
        e.set_ordering(N.PDGB_ORDER_DENSE)
        _against_oracle(e, body, params, 3)


# Sparse trees: small and tiny supernodes beside tiles, one level and several;
# odd and even iteration counts (the two y buffers), with and without the
# convergence test and refinement.
@pytest.mark.parametrize("dims,iters,tol,refine", [((2, 1, 1), 1, 0.0, 0), ((4, 3, 5), 3, 0.0, 0), ((6, 5, 7), 4, 0.0, 1),
                                                   ((9, 4, 6), 5, 0.0, 2), ((9, 9, 9), 5, 1e-4, 0),
                                                   ((9, 9, 9), 5, 1e-4, 1), ((3, 17, 5), 2, 0.0, 3)])
def test_sparse_solve_over_forms(dims, iters, tol, refine):
    body = mesh.make_grid_body(*dims, young=3e5, jitter=0.1, seed=2)
    params = SolverParams(num_iterations=iters, tol=tol, solver=1, refine_steps=refine)
    with PdSolver(body, params) as e:
        _against_oracle(e, body, params, 4)


# The product with the root's inverse: up to 1,024 pivots, 8 rows a CTA; the
# whole solve (two right-hand sides in turn) or above one or two levels; odd and
# even iteration counts, the convergence test, refinement.
@pytest.mark.parametrize("dims,order,iters,tol,refine", [((1, 1, 1), 2, 1, 0.0, 0), ((1, 4, 6), 2, 2, 0.0, 1),
                                                         ((16, 9, 5), 2, 3, 0.0, 0), ((15, 7, 7), 2, 4, 0.0, 0),
                                                         ((18, 8, 5), 2, 3, 0.0, 0), ((6, 6, 6), 0, 3, 1e-4, 2),
                                                         ((10, 10, 10), 0, 3, 0.0, 2), ((10, 10, 10), 0, 4, 1e-4, 0),
                                                         ((31, 2, 29), 0, 5, 0.0, 1)])
def test_root_product_over_forms(dims, order, iters, tol, refine):
    body = mesh.make_grid_body(*dims, young=1e5, jitter=0.1, seed=13)
    params = SolverParams(num_iterations=iters, tol=tol, solver=1, refine_steps=refine)
    with PdSolver(body, params) as e:
        e.set_ordering(order)
        _against_oracle(e, body, params, 3)


@pytest.mark.parametrize("mode", [N.PDGB_SOLVE_CTA, N.PDGB_SOLVE_CLUSTER, N.PDGB_SOLVE_LEVELS, N.PDGB_SOLVE_PERSISTENT])
def test_batch_of_uneven_trees(mode):
    """Trees of different heights share the levels' launches."""
    bodies = [mesh.make_grid_body(*d, young=1e5, jitter=0.1, seed=i) for i, d in
              enumerate([(1, 1, 1), (8, 8, 8), (2, 2, 2), (4, 13, 3), (3, 3, 4)])]
    params = SolverParams(num_iterations=5, solver=1)
    with PdSolver(bodies, params) as e:
        e.set_solve_mode(mode)
        e.update(3)
        for b, body in enumerate(bodies):
            X, _ = e.download_body(b)
            Xo, _, _ = O.simulate(body, params, 3, precision=64)
            assert rel_l2(X, Xo) < TOL, b


# Panels of 32 pivots: below, at and past one and two of them, odd remainders,
# rows below the pivots (sparse) and none (dense).
@pytest.mark.parametrize("dims,order", [((1, 1, 6), 2), ((1, 1, 7), 2), ((1, 2, 5), 2), ((3, 3, 3), 2), ((1, 4, 12), 2),
                                        ((4, 4, 4), 2), ((7, 6, 5), 0), ((10, 3, 8), 0), ((9, 9, 8), 2)])
def test_gpu_factor_at_panel_edges(dims, order):
    body = mesh.make_grid_body(*dims, young=1e5, jitter=0.1, seed=9)
    blocks = []
    for dev in (N.PDGB_FACTOR_GPU, N.PDGB_FACTOR_HOST):
        with PdSolver(body, SolverParams(num_iterations=2, solver=1)) as e:
            e.set_ordering(order)
            e.set_factor_device(dev)
            e.prepare()
            blocks.append(e.factor_blocks())
    g, h = blocks
    # both round an FP64 result of relative error ~1e-13 to float: the same, or
    # neighbours where it lies near a midpoint
    assert np.all(np.abs(g - h) <= np.spacing(np.abs(h)) + 1e-12 * np.abs(h).max())
    assert np.mean(g != h) < 1e-3


# Threads a CTA of the allocation-free step change at 152 x 256 and 152 x 512
# tets; 131,072 tets and 32,768 vertices are the most.
@pytest.mark.parametrize("dims,dbc", [((1, 1, 1), True), ((1, 3, 17), False), ((20, 19, 20), True), ((20, 20, 20), True),
                                      ((25, 25, 25), True), ((29, 30, 30), True)])
def test_noalloc_launch_shapes(dims, dbc):
    torch = pytest.importorskip("torch")
    lib = N.lib()
    body = mesh.make_grid_body(*dims, young=2e5, jitter=0.1, seed=12, pin="top" if dbc else None)
    params = SolverParams(num_iterations=13, rho=0.9995, solver=0)
    dev = {k: torch.from_numpy(np.ascontiguousarray(getattr(body, k))).cuda() for k in ("X", "tets", "mass", "mu", "dbc")}
    m = N.pdgb_noalloc_mesh(body.num_verts, body.num_tets, dev["tets"].data_ptr(), dev["X"].data_ptr(),
                            dev["mass"].data_ptr(), dev["mu"].data_ptr(), dev["dbc"].data_ptr() if dbc else None)
    X, V = dev["X"].clone(), torch.zeros_like(dev["X"])
    prm = params.to_c()
    for steps in (0, 2):
        st = lib.pdgb_step_noalloc(C.byref(m), C.byref(prm), X.data_ptr(), V.data_ptr(), steps,
                                   torch.cuda.current_stream().cuda_stream)
        assert st == N.PDGB_OK
        if steps == 0:
            assert torch.equal(X, dev["X"])
    Xo, _, _ = O.simulate(body, params, 2, precision=64)
    assert rel_l2(X.cpu().numpy(), Xo) < TOL


def test_noalloc_more_steps_than_one_launch_holds():
    torch = pytest.importorskip("torch")
    lib = N.lib()
    body = mesh.make_grid_body(2, 2, 2, young=2e5, jitter=0.1, seed=1)
    params = SolverParams(num_iterations=2048, rho=0.9, solver=0)  # 4 steps a launch
    dev = {k: torch.from_numpy(np.ascontiguousarray(getattr(body, k))).cuda() for k in ("X", "tets", "mass", "mu", "dbc")}
    m = N.pdgb_noalloc_mesh(body.num_verts, body.num_tets, dev["tets"].data_ptr(), dev["X"].data_ptr(),
                            dev["mass"].data_ptr(), dev["mu"].data_ptr(), dev["dbc"].data_ptr())
    X, V = dev["X"].clone(), torch.zeros_like(dev["X"])
    prm = params.to_c()
    assert lib.pdgb_step_noalloc(C.byref(m), C.byref(prm), X.data_ptr(), V.data_ptr(), 6, None) == N.PDGB_OK
    torch.cuda.synchronize()
    Xo, _, _ = O.simulate(body, params, 6, precision=64)
    assert rel_l2(X.cpu().numpy(), Xo) < TOL


# Iterations 10 and 11 are where the iterate buffers begin to take turns and
# prev is first read; tets on both sides of the default tile sizes' limits.
@pytest.mark.parametrize("iters", [1, 2, 10, 11, 12, 13, 20])
def test_jacobi_iterate_buffers(iters):
    body = mesh.make_grid_body(5, 4, 6, young=2e5, jitter=0.1, seed=4)
    params = SolverParams(num_iterations=iters, rho=0.9995, solver=0)
    with PdSolver(body, params) as e:
        _against_oracle(e, body, params, 3)


@pytest.mark.parametrize("dims", [(16, 16, 15), (16, 16, 16), (28, 28, 28), (28, 28, 29)])
def test_jacobi_at_the_default_tile_limits(dims):
    body = mesh.make_grid_body(*dims, young=1e6, poisson=0.45, jitter=0.1, seed=4)
    params = SolverParams(num_iterations=12, rho=0.9995, solver=0)
    with PdSolver(body, params) as e:
        _against_oracle(e, body, params, 1)


# Scenes whose cubics have far roots (Newton iterates that swap between two
# floats) and distances around the float thresholds: small, ordinary and large
# coordinates, and offsets that leave few bits for the differences.
@pytest.mark.parametrize("scale,offset", [(1e-3, 0.0), (1.0, 0.0), (60.0, 0.0), (1.0, 90.0), (4e3, 0.0)])
def test_collision_query_over_scales(scale, offset):
    rng = np.random.default_rng(17)
    nb, per = 3, 120
    cent = rng.uniform(-0.4, 0.4, (nb * per, 1, 3))
    X = ((cent + rng.uniform(-0.06, 0.06, (nb * per, 3, 3))).reshape(-1, 3) * scale + offset).astype(np.float32)
    XT = (X + rng.uniform(-0.08, 0.08, X.shape) * scale).astype(np.float32)
    XT[: 30] = X[: 30]  # some do not move at all
    tris = np.arange(X.shape[0], dtype=np.uint32).reshape(-1, 3)
    body = np.repeat(np.arange(nb, dtype=np.int32), per)
    tI, nrm, info = ccd_detect(tris, body, X, XT)
    tIo, nrmo, (pairs, _, marked) = O.ccd_detect(tris, body, X, XT)
    assert info["candidate_pairs"] == pairs and info["vertices_hit"] == marked
    assert np.array_equal(tI, tIo)  # the same decisions
    assert np.abs(nrm - nrmo).max() <= 1e-6


def _soup(n, bodies, seed, size=0.06, speed=0.08, room=0.5, stretch=1.0):
    rng = np.random.default_rng(seed)
    cent = rng.uniform(-room, room, (n, 1, 3))
    X = cent + rng.uniform(-size, size, (n, 3, 3)) * np.array([stretch, 1.0, 1.0])
    X = X.reshape(-1, 3).astype(np.float32)
    XT = (X + rng.uniform(-speed, speed, X.shape)).astype(np.float32)
    tris = np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    return tris, rng.integers(0, bodies, n).astype(np.int32), X, XT


# Groups of 32 triangles and tree levels of 32: one triangle, at and past one
# group, one and two levels, three; the lists that grow (every box over every
# other: 561 group pairs past 528, pairs past 16 a triangle); slivers a hundredth
# as wide as long, far from the origin; hardly moving and fast ones.
@pytest.mark.parametrize("n,bodies,kw", [(1, 1, {}), (2, 2, {"room": 0.02}), (31, 3, {"room": 0.1}), (32, 2, {"room": 0.1}),
                                         (33, 2, {"room": 0.1}), (1024, 5, {"room": 0.7}), (1025, 40, {"room": 0.7}),
                                         (1056, 2, {"room": 0.01, "size": 0.3}), (33000, 300, {"room": 4.0}),
                                         (600, 4, {"stretch": 100.0, "size": 0.01}),
                                         (600, 4, {"speed": 1e-4, "room": 0.15}), (600, 4, {"speed": 3.0})])
def test_collision_tree_and_lists(n, bodies, kw):
    tris, body, X, XT = _soup(n, bodies, 40 + n % 17, **kw)
    if kw.get("stretch"):
        X, XT = X + np.float32(20.0), XT + np.float32(20.0)
    if n == 1025:  # triangles of different bodies that share vertices
        tris[1:400:2, 0] = tris[0:400:2, 1][:200]
    tI, nrm, info = ccd_detect(tris, body, X, XT)
    tIo, nrmo, (pairs, _, marked) = O.ccd_detect(tris, body, X, XT)
    assert info["candidate_pairs"] == pairs and info["vertices_hit"] == marked
    assert np.array_equal(tI, tIo)  # the same float operations decide both
    assert np.abs(nrm - nrmo).max() <= 1e-6
    if n == 1056:
        assert info["regrows"] == 1


# The closed form and the squarings meet where det F = 0.06 |F|^3, for a whole
# warp: strains up to there and past it, flat and inverted elements, scales down
# to where squares leave float's range.  Both round a result of condition
# |F| / (s2 + s3), at most 4 here: some ten units of 6e-8 times that.
@pytest.mark.parametrize("strain", [0.0, 0.01, 0.3, 1.0])
@pytest.mark.parametrize("scale", [1e-12, 1e-4, 1.0, 1e4, 1e12])
def test_rotation_over_strains_and_scales(strain, scale):
    rng = np.random.default_rng(5)
    n = 4000
    U, V = (np.linalg.qr(rng.normal(size=(n, 3, 3)))[0] for _ in range(2))
    U *= np.sign(np.linalg.det(U))[:, None, None]
    V *= np.sign(np.linalg.det(V))[:, None, None]
    s = 1.0 + strain * rng.normal(size=(n, 3))
    s[: n // 8, 2] = 0.0
    s[n // 8: n // 4, 2] = -0.3
    F = np.einsum("nij,nj,nkj->nik", U, s, V).astype(np.float32)
    Fd = F.astype(np.float64)
    u, sv, vt = np.linalg.svd(Fd)
    sign = np.sign(np.linalg.det(u @ vt))
    D = np.ones((n, 3))
    D[:, 2] = sign
    R = np.einsum("nij,nj,njk->nik", u, D, vt)
    well = sv[:, 1] + sign * sv[:, 2] > 0.25 * np.linalg.norm(sv, axis=1)
    assert well.mean() > 0.5
    F = np.ascontiguousarray(F * np.float32(scale))
    out = np.empty_like(F)
    N.check(N.lib().pdgb_closest_rotations(n, F.ctypes.data, out.ctypes.data, N.PDGB_ROTATION_QUAT), "rotations")
    err = np.abs(out - R).max(axis=(1, 2))[well]
    assert err.max() < 4 * 10 * 6e-8 and np.sqrt(np.mean(err ** 2)) < 6e-7
