"""The work that a program has this engine do, as measurable cases.

A case is one pass through the public entry points: the state goes in, the
engine advances it by the frame's time steps, the state comes out.  The sizes,
materials and iteration counts are those of the named workloads in
``pdgb.mesh``, of the tests and of ``bench.py``, and ragged ones between them.

listed() the cases; draw(rng) more of the same ranges; prepare(case, seed) the
bodies, the engine and the state arrays a program has in hand; run(state) one
pass; work(case) the bytes and operations it cannot do without; exact(case,
seed) the same step in 64 bits, in plain torch.
"""
import ctypes as C
import math
import sys
import time
from pathlib import Path

import numpy as np
import torch

_PKG = Path(__file__).resolve().parent.parent / "soft-body-simulation-cuda_gb300"
if str(_PKG) not in sys.path:
    sys.path.insert(0, str(_PKG))

import pdgb  # noqa: E402
from pdgb import PdServer, PdSolver, SolverParams, _native as N, mesh, meshio, scene  # noqa: E402

DT = 1.0 / 120.0


def listed():
    return [
        # An interactive viewer's body held by the mouse: a few hundred vertices,
        # state read and written by the host every frame of two steps.
        {"name": "drag_small", "kind": "jacobi", "nx": 8, "ny": 6, "nz": 5, "iters": 20, "rho": 0.9995, "steps": 2,
         "drag": True, "host": True},
        # A thin sheet with the default parameters, ragged in every direction.
        {"name": "jacobi_sheet", "kind": "jacobi", "nx": 47, "ny": 5, "nz": 61, "iters": 10, "rho": 0.9992, "steps": 2,
         "drag": False, "host": False},
        # The large Jacobi + Chebyshev cube of the benchmark (1.3 M tets), one step.
        {"name": "jacobi_cube64", "kind": "jacobi", "nx": 64, "ny": 64, "nz": 64, "iters": 20, "rho": 0.9995,
         "steps": 1, "drag": False, "host": False},
        # A body whose working set is past the L2 cache (2.0 M tets), odd dimensions.
        {"name": "jacobi_past_l2", "kind": "jacobi", "nx": 79, "ny": 61, "nz": 83, "iters": 20, "rho": 0.9995,
         "steps": 1, "drag": False, "host": False},
        # The small Cholesky cube as its tuned configuration runs it (one dense
        # supernode, 128-tet tiles), state on the host.
        {"name": "chol_cube10", "kind": "cholesky", "nx": 10, "ny": 10, "nz": 10, "iters": 10, "refine": 0, "steps": 2,
         "hetero": False, "order": "dense", "tile": 128, "host": True},
        # A mid-size ragged body with FP64-residual refinement, as a program that
        # wants the last digits runs it; engine defaults otherwise.
        {"name": "chol_refined", "kind": "cholesky", "nx": 19, "ny": 11, "nz": 23, "iters": 10, "refine": 2,
         "steps": 2, "hetero": False, "order": "amd", "tile": 512, "host": False},
        # The heterogeneous 40^3 cube of the precision workload (320 k tets).
        {"name": "chol_cube40", "kind": "cholesky", "nx": 40, "ny": 40, "nz": 40, "iters": 10, "refine": 0, "steps": 1,
         "hetero": True, "order": "amd", "tile": 512, "host": False},
        # Many uneven bodies in one engine, 4..24 cells per axis: the batching workload.
        {"name": "batch_chol", "kind": "batch", "bodies": 128, "lo": 4, "hi": 24, "solver": "cholesky", "iters": 10,
         "steps": 1},
        # Bodies dropped on one another and onto a floor, collision handling on, as
        # the reference's scenes run by default.
        {"name": "contact_scene", "kind": "contact", "bodies": 8, "lo": 6, "hi": 12, "iters": 20, "steps": 2},
        # A burst of scene requests through the server, from submission to the last
        # result: sizes log-uniform from 1e3 tets up, each with its own step count.
        {"name": "serve_jacobi", "kind": "serve", "requests": 24, "top": 300000, "solver": "jacobi", "most": 16},
        {"name": "serve_chol", "kind": "serve", "requests": 12, "top": 100000, "solver": "cholesky", "most": 16},
        # A plugin that may not allocate: device pointers in, two steps, out.
        {"name": "noalloc_block", "kind": "noalloc", "nx": 12, "ny": 9, "nz": 10, "iters": 20, "rho": 0.9995,
         "steps": 2},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def dims(lo, hi):
        """Ragged box of log-uniform tet count lo..hi, aspect up to 4."""
        cells = math.exp(rng.uniform(math.log(lo), math.log(hi))) / 5.0
        a, b = math.exp(rng.uniform(-0.7, 0.7)), math.exp(rng.uniform(-0.7, 0.7))
        base = cells ** (1.0 / 3.0)
        nx, ny = max(1, round(base * a)), max(1, round(base * b))
        return nx, ny, max(1, int(cells / (nx * ny)))

    kind = rng.choice(["jacobi", "jacobi", "cholesky", "cholesky", "batch", "contact", "serve", "noalloc"])
    if kind == "jacobi":
        nx, ny, nz = dims(600, 1.9e6)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "iters": rng.choice([7, 10, 12, 20]),
                "rho": rng.choice([0.9992, 0.9995]), "steps": rng.choice([1, 2]), "drag": nx * ny * nz < 4000,
                "host": rng.random() < 0.3}
    if kind == "cholesky":
        nx, ny, nz = dims(600, 2.4e5)
        small = (nx + 1) * (ny + 1) * (nz + 1) <= 1800
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "iters": rng.choice([5, 10]),
                "refine": rng.choice([0, 0, 1, 2]) if 5 * nx * ny * nz < 60000 else 0, "steps": rng.choice([1, 2]),
                "hetero": rng.random() < 0.5, "order": "dense" if small and rng.random() < 0.5 else "amd",
                "tile": rng.choice([128, 512]), "host": rng.random() < 0.3}
    if kind == "batch":
        return {"kind": kind, "bodies": log_int(2, 80), "lo": rng.randint(2, 5), "hi": rng.randint(8, 24),
                "solver": rng.choice(["cholesky", "cholesky", "jacobi"]), "iters": rng.choice([5, 10]), "steps": 1}
    if kind == "contact":
        return {"kind": kind, "bodies": rng.randint(2, 8), "lo": rng.randint(3, 6), "hi": rng.randint(7, 12),
                "iters": rng.choice([10, 20]), "steps": rng.choice([1, 2])}
    if kind == "serve":
        solver = rng.choice(["jacobi", "cholesky"])
        return {"kind": kind, "requests": rng.randint(3, 12), "top": log_int(5e3, 1e5), "solver": solver,
                "most": rng.randint(4, 16)}
    nx, ny, nz = dims(600, 1.2e5)
    return {"kind": "noalloc", "nx": nx, "ny": ny, "nz": nz, "iters": rng.choice([10, 20]), "rho": 0.9995,
            "steps": rng.choice([1, 2])}


# ------------------------------------------------------------------ inputs
_SPLIT = (((1, 0, 3, 5), (2, 0, 3, 6), (4, 0, 5, 6), (7, 3, 6, 5), (0, 3, 5, 6)),
          ((0, 1, 2, 4), (3, 1, 2, 7), (5, 1, 4, 7), (6, 2, 4, 7), (1, 2, 4, 7)))


def _grid(nx, ny, nz, cell, rng, jitter=0.1, young=1e6, poisson=0.45, density=1000.0, pin=True, origin=(0.0, 0.0, 0.0)):
    """A jittered hex grid of 5 tets per cell, as plain arrays."""
    vid = np.arange((nx + 1) * (ny + 1) * (nz + 1), dtype=np.int64)
    i, j, k = vid % (nx + 1), (vid // (nx + 1)) % (ny + 1), vid // ((nx + 1) * (ny + 1))
    X = np.stack([i, j, k], 1).astype(np.float64)
    X += rng.uniform(-jitter, jitter, X.shape)
    X = (X * np.asarray(cell) + np.asarray(origin)).astype(np.float32)
    cells = np.arange(nx * ny * nz, dtype=np.int64)
    ci, cj, ck = cells % nx, (cells // nx) % ny, cells // (nx * ny)
    first = ci + (nx + 1) * (cj + (ny + 1) * ck)
    step = np.array([1, nx + 1, (nx + 1) * (ny + 1)])
    odd = ((ci + cj + ck) & 1).astype(bool)
    tets = np.empty((cells.size, 5, 4), np.int64)
    for parity, split in enumerate(_SPLIT):
        off = np.array([[sum(step[d] for d in range(3) if c >> d & 1) for c in t] for t in split])
        at = np.nonzero(odd == bool(parity))[0]
        tets[at] = first[at, None, None] + off[None]
    tets = tets.reshape(-1, 4)
    x = X.astype(np.float64)
    e = [x[tets[:, c]] - x[tets[:, 0]] for c in (1, 2, 3)]
    vol = np.einsum("ij,ij->i", np.cross(e[0], e[1]), e[2]) / 6.0
    neg = vol < 0
    tets[neg, 2], tets[neg, 3] = tets[neg, 3].copy(), tets[neg, 2].copy()
    m = np.abs(vol) * density / 4.0
    mass = sum(np.bincount(tets[:, c], weights=m, minlength=vid.size) for c in range(4))
    mu = np.broadcast_to(np.asarray(young, np.float64) / (2.0 * (1.0 + np.asarray(poisson, np.float64))), vol.shape)
    dbc = (j == ny).astype(np.float32) if pin else np.zeros(vid.size, np.float32)
    return {"X0": X, "tets": tets.astype(np.uint32), "mass": mass.astype(np.float32), "mu": mu.astype(np.float32),
            "dbc": dbc}


def _moving(body, rng, speed=2.0, bend=0.01):
    """A body in mid-motion: smooth velocities of some m/s, strains of a few percent."""
    x = body["X0"].astype(np.float64)
    span = np.maximum(x.max(0) - x.min(0), 1e-6)
    u = (x - x.min(0)) / span
    a, ph = rng.uniform(0.5, 2.5, (3, 3)), rng.uniform(0, 2 * math.pi, (3, 3))
    free = (1.0 - u[:, 1:2]) * (body["dbc"] == 0)[:, None] if body["dbc"].any() else 1.0  # nothing moves at the pins
    V = sum(np.sin(u[:, [d]] * a[d] + ph[d]) for d in range(3)) * speed
    b = sum(np.cos(u[:, [d]] * a[d] * 2.0 + ph[d]) for d in range(3)) * bend * span.min()
    return (x + b * free).astype(np.float32), (V * free).astype(np.float32)


def _single(case, seed):
    rng = np.random.default_rng([seed, case["nx"], case["ny"], case["nz"]])
    n = (case["nx"], case["ny"], case["nz"])
    if case.get("hetero"):
        nt = 5 * n[0] * n[1] * n[2]
        E = np.exp(rng.uniform(math.log(1e4), math.log(1e7), nt))
        nu = rng.uniform(0.3, 0.45, nt)
    else:
        E, nu = (1e5, 0.4) if case["kind"] == "cholesky" else (1e6, 0.45)
    body = _grid(*n, 1.0 / max(n), rng, young=E, poisson=nu)
    body["X"], body["V"] = _moving(body, rng)
    return body


def _uneven(rng, nx, ny, nz, **more):
    """A body of the batching workload's materials, 1/16 m cells."""
    return _grid(nx, ny, nz, 1.0 / 16.0, rng, jitter=0.05, young=math.exp(rng.uniform(math.log(1e4), math.log(1e7))),
                 poisson=rng.uniform(0.3, 0.45), density=rng.uniform(800.0, 1200.0), **more)


def _bodies(case, seed):
    """Sizes and step counts come from the case, materials and motion from the seed."""
    rng = np.random.default_rng([seed, 7])
    shape = np.random.default_rng([case.get("bodies", 0), case.get("requests", 0), case.get("lo", 0), case.get("top", 0)])
    out = []
    if case["kind"] == "batch":
        for _ in range(case["bodies"]):
            b = _uneven(rng, *(int(v) for v in shape.integers(case["lo"], case["hi"] + 1, 3)))
            b["X"], b["V"] = _moving(b, rng)
            out.append(b)
    elif case["kind"] == "serve":
        for q in range(case["requests"]):
            t = math.exp(math.log(1e3) + math.log(case["top"] / 1e3) * (q + shape.uniform(0, 1)) / case["requests"])
            n = max(1, int((t / 5.0) ** (1.0 / 3.0)))
            b = _uneven(rng, n, n, max(1, round(t / (5.0 * n * n))))
            b["X"], b["V"], b["steps"] = b["X0"], _moving(b, rng)[1], int(shape.integers(4, case["most"] + 1))
            out.append(b)
    else:
        # pairs: one body falls onto another, which falls onto the floor y = 0
        for q in range(case["bodies"]):
            n = [int(v) for v in shape.integers(case["lo"], case["hi"] + 1, 3)]
            top = q % 2 == 1 and q > 0
            below = out[q - 1] if top else None
            base = float(below["X0"][:, 1].max()) + 0.012 if top else 0.02
            b = _uneven(rng, *n, pin=False, origin=(2.0 * (q // 2), base, 0.01 * q))
            b["X"], b["V"] = b["X0"], np.zeros_like(b["X0"])
            b["V"][:, 1] = -(5.0 + rng.uniform(0, 1) if top else 1.0 + rng.uniform(0, 1))
            out.append(b)
    return out


# ----------------------------------------------------------------- prepare
_ONE_STREAM = []


def _stream():
    """The program's one compute stream, which all its engines share."""
    if not _ONE_STREAM:
        _ONE_STREAM.append(torch.cuda.Stream())
    return _ONE_STREAM[0].cuda_stream


def _soft(b):
    return mesh.SoftBody(X=b["X0"], tets=b["tets"], mass=b["mass"], mu=b["mu"], dbc=b["dbc"], V=b["V"])


def _params(case):
    chol = case.get("solver", case["kind"]) == "cholesky"
    return SolverParams(num_iterations=case.get("iters", 10), rho=case.get("rho", 0.9995), solver=1 if chol else 0,
                        refine_steps=case.get("refine", 0))


def _cat(bodies, key):
    return np.concatenate([b[key] for b in bodies])


def prepare(case, seed):
    kind = case["kind"]
    prm = _params(case)
    if kind == "serve":
        # the server keeps no meshes: a stream of scenes that do not come twice
        return {"kind": kind, "server": PdServer(prm, hbm_budget_bytes=16 << 30, cache_entries=-1, stream=_stream()),
                "requests": [(_soft(b), b["steps"]) for b in _bodies(case, seed)]}
    if kind == "noalloc":
        b = _single(case, seed)
        s = {k: torch.from_numpy(b[k].view(np.int32) if k == "tets" else b[k]).cuda()
             for k in ("X0", "tets", "mass", "mu", "dbc", "X", "V")}
        s["mesh"] = N.pdgb_noalloc_mesh(b["X0"].shape[0], b["tets"].shape[0], s["tets"].data_ptr(), s["X0"].data_ptr(),
                                        s["mass"].data_ptr(), s["mu"].data_ptr(), s["dbc"].data_ptr())
        s.update(kind=kind, prm=prm.to_c(), steps=case["steps"], oX=torch.empty_like(s["X"]), oV=torch.empty_like(s["V"]))
        return s
    if kind in ("batch", "contact"):
        bodies = _bodies(case, seed)
        eng = PdSolver([_soft(b) for b in bodies], prm, stream=_stream())
        X, V = _cat(bodies, "X"), _cat(bodies, "V")
    else:
        b = _single(case, seed)
        eng = PdSolver(_soft(b), prm, stream=_stream())
        X, V = b["X"], b["V"]
    s = {"kind": kind, "eng": eng, "steps": case["steps"], "host": case.get("host", False)}
    if kind == "cholesky":
        eng.set_ordering({"amd": N.PDGB_ORDER_AMD, "dense": N.PDGB_ORDER_DENSE}[case["order"]])
        eng.set_tile_size(case["tile"])
    if kind == "contact":
        off = np.cumsum([0] + [b["X0"].shape[0] for b in bodies])
        eng.set_collision_surface(np.concatenate([meshio.surface_triangles(b["tets"]) + np.uint32(o)
                                                  for b, o in zip(bodies, off)]))
        eng.set_fixed_bodies([scene.plane((0.0, 0.0, 0.0))])
        eng.enable_collision(True)
    if case.get("drag"):
        at, w, off, s["target"] = _drag(b)
        eng.set_drag(w, off)
        eng.set_drag_target(s["target"])
    eng.prepare()
    if s["host"]:
        s["X"], s["V"] = X, V
    else:
        s["X"], s["V"] = torch.from_numpy(X).cuda(), torch.from_numpy(V).cuda()
        s["oX"], s["oV"] = torch.empty_like(s["X"]), torch.empty_like(s["V"])
        s["oXT"] = torch.empty_like(s["X"]) if kind == "contact" else None
    return s


def _drag(b):
    """The grabbed vertex, weights 10 on the vertices near it, offsets and target."""
    free = np.nonzero(b["dbc"] == 0)[0]
    at = int(free[np.argmax(b["X"][free, 0] - b["X"][free, 1])])
    d = b["X"].astype(np.float64) - b["X"][at].astype(np.float64)
    w = np.where(((d * d).sum(1) < 0.03) & (b["dbc"] == 0), 10.0, 0.0).astype(np.float32)
    return at, w, d.astype(np.float32), (b["X"][at] + np.array([0.05, -0.02, 0.03], np.float32)).astype(np.float32)


# --------------------------------------------------------------------- run
def run(s):
    lib = N.lib()
    if s["kind"] == "serve":
        srv = s["server"]
        ids = [srv.submit(body, k) for body, k in s["requests"]]
        done0 = srv.stats()
        last = done0["completed"] + done0["failed"] + len(ids)
        while True:
            active, _ = srv.tick()
            st = srv.stats()
            if st["completed"] + st["failed"] >= last:
                break
            if active == 0 and st["finishing"] == 0 and st["ready"] == 0:
                time.sleep(0.0001)  # the layout workers have the next request
        got = [srv.result(r) for r in ids]
        return {"X": np.concatenate([g[0] for g in got]), "V": np.concatenate([g[1] for g in got])}
    if s["kind"] == "noalloc":
        s["oX"].copy_(s["X"])
        s["oV"].copy_(s["V"])
        N.check(lib.pdgb_step_noalloc(C.byref(s["mesh"]), C.byref(s["prm"]), s["oX"].data_ptr(), s["oV"].data_ptr(),
                                      s["steps"], torch.cuda.current_stream().cuda_stream), "pdgb_step_noalloc")
        return {"X": s["oX"], "V": s["oV"]}
    eng = s["eng"]
    if s["host"]:
        if "target" in s:
            eng.set_drag_target(s["target"])
        eng.upload_state(s["X"], s["V"])
        eng.update(s["steps"])
        X, V = eng.download_state()
        return {"X": X, "V": V}
    h, dev = eng.handle, N.PDGB_MEM_DEVICE
    if "target" in s:
        eng.set_drag_target(s["target"])
    N.check(lib.pdgb_upload_state(h, s["X"].data_ptr(), s["V"].data_ptr(), dev), "pdgb_upload_state")
    eng.update(s["steps"])
    N.check(lib.pdgb_download_state(h, s["oX"].data_ptr(), s["oV"].data_ptr(), dev), "pdgb_download_state")
    out = {"X": s["oX"], "V": s["oV"]}
    if s["oXT"] is not None:
        N.check(lib.pdgb_download_xtilde(h, s["oXT"].data_ptr(), dev), "pdgb_download_xtilde")
        out["XT"] = s["oXT"]
    return out


# -------------------------------------------------------------------- work
def work(case):
    """Per iteration: 56 bytes a tet (four ids, nine floats of DmInv, the weight)
    and 68 a vertex for a fused Jacobi iteration, 36 and the factor's nonzeros
    (a value and an index each, forward and backward) with Cholesky; 48 bytes a
    vertex in and out.  About 480 operations a tet (deformation gradient, closest
    rotation, corner forces), 12 a nonzero of the factor."""
    sizes, steps = _sizes(case), case.get("steps", 1)
    by = fl = 0.0
    for nt, nv, st in sizes:
        st = st or steps
        it = case.get("iters", 10) * st
        if case.get("solver", case["kind"]) == "cholesky":
            nnz = 48268.0 * (nv / 1331.0) ** 1.578  # measured nonzeros of 11^3 and 41^3 vertex grids
            by += it * (56.0 * nt + 36.0 * nv + (1 + case.get("refine", 0)) * (16.0 * nnz + 68.0 * nv))
            fl += it * (480.0 * nt + (1 + case.get("refine", 0)) * 12.0 * nnz)
        else:
            by += it * (56.0 * nt + 68.0 * nv)
            fl += it * 480.0 * nt
        by += 48.0 * nv
    return {"bytes": by, "flops": fl}


def _sizes(case):
    """(tets, vertices, steps or 0) of each body; drawn sizes by their means."""
    if "nx" in case:
        n = (case["nx"], case["ny"], case["nz"])
        return [(5 * n[0] * n[1] * n[2], (n[0] + 1) * (n[1] + 1) * (n[2] + 1), 0)]
    if case["kind"] == "serve":
        out = []
        for q in range(case["requests"]):
            t = math.exp(math.log(1e3) + math.log(case["top"] / 1e3) * (q + 0.5) / case["requests"])
            out.append((t, ((t / 5.0) ** (1.0 / 3.0) + 1) ** 3, (4 + case["most"]) / 2.0))
        return out
    m = (case["lo"] + case["hi"]) / 2.0
    return [(5 * m ** 3, (m + 1) ** 3, 0)] * case["bodies"]


# ------------------------------------------------------------------- exact
def exact(case, seed):
    """The PD iteration in 64 bits: closest rotations by Newton's polar iteration or an SVD,
    K x = b by conjugate gradients to 1e-13."""
    if case["kind"] == "contact":
        return None  # which vertices touch is decided by float comparisons
    if case["kind"] in ("batch", "serve"):
        bodies = _bodies(case, seed)
        off = np.cumsum([0] + [b["X0"].shape[0] for b in bodies])
        sys_ = {k: _cat(bodies, k) for k in ("X0", "mass", "mu", "dbc", "X", "V")}
        sys_["tets"] = np.concatenate([b["tets"] + np.uint32(o) for b, o in zip(bodies, off)])
        wanted = np.concatenate([np.full(b["X0"].shape[0], b.get("steps", case.get("steps", 0))) for b in bodies])
    else:
        sys_ = _single(case, seed)
        wanted = np.full(sys_["X0"].shape[0], case["steps"])
    prm = _params(case)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = {"dtype": torch.float64, "device": dev}

    def put(a):
        return torch.from_numpy(np.asarray(a, np.float64)).to(dev)

    X0, x, v, m, pin = (put(sys_[k]) for k in ("X0", "X", "V", "mass", "dbc"))
    T = torch.from_numpy(sys_["tets"].astype(np.int64)).to(dev)
    nv, nt = X0.shape[0], T.shape[0]
    dt, g, pw = float(np.float32(prm.dt)), float(np.float32(prm.gravity)), float(prm.positional_weight)
    Dm = torch.stack([X0[T[:, c]] - X0[T[:, 0]] for c in (1, 2, 3)], 2)  # columns are edges
    inv, det = _adjugate(Dm)
    inv = inv / det[:, None, None]
    c = det.abs() / 6.0 * put(sys_["mu"])
    B = torch.cat([-(inv.sum(1, keepdim=True)), inv], 1)  # [nt, corner, 3]: rows of G^T DmInv
    pinned = (pin > 0)[:, None]
    mdt2 = ((m + pin * pw) / (dt * dt))[:, None]
    diag = torch.zeros(nv, **f64)
    BB = c[:, None, None] * (B @ B.transpose(1, 2))
    for j in range(4):
        diag.index_add_(0, T[:, j], BB[:, j, j])
    diag = diag[:, None]
    pin_rhs = X0 * (pw / (dt * dt))
    w = torch.zeros(nv, 1, **f64)
    if case.get("drag"):
        _, wd, off, target = _drag(sys_)
        w, goal = put(wd)[:, None], put(target)[None] + put(off)
    held = w > 0
    chol = prm.solver == 1
    K = _system(T, BB, mdt2[:, 0], nv, dev) if chol else None
    outX, outV = x.clone(), v.clone()
    left = torch.from_numpy(wanted).to(dev)
    for step in range(1, int(wanted.max()) + 1):
        grav = torch.zeros(nv, 3, **f64)
        grav[:, 1] = -g * m / mdt2[:, 0]
        s = x + dt * v + grav
        base_m = mdt2
        if case.get("drag"):
            s = torch.where(held, goal, s)
            base_m = torch.where(held & ~pinned, (m[:, None] + w) / (dt * dt), mdt2)
        base = base_m * s
        if case.get("drag") and bool(pinned.any()):
            base = torch.where(held & ~pinned, s * w, base)
        prev, omega = s, 1.0
        for i in range(prm.num_iterations):
            omega = 1.0 if i <= 10 else 2.0 / (2.0 - prm.rho ** 2) if i == 11 else 4.0 / (4.0 - prm.rho ** 2 * omega)
            F = torch.stack([s[T[:, k]] - s[T[:, 0]] for k in (1, 2, 3)], 2) @ inv
            R = _polar(F)
            M = c[:, None, None] * (B @ (R if chol else R - F).transpose(1, 2))  # [nt, corner, 3]
            b = base.clone()
            for k in range(4):
                b.index_add_(0, T[:, k], M[:, k])
            b = torch.where(pinned, pin_rhs, b)
            if chol:
                s = _cg(K, diag + mdt2, b, s)
                continue
            nx = torch.where(held, s, (b - mdt2 * s) / (mdt2 + diag) + s)
            nx = 0.9 * (nx - s) + s
            if i >= 11:
                nx = (nx - prev) * omega + prev
            prev, s = s, nx
        v = torch.where(held, torch.zeros_like(s), (s - x) / dt)
        x = s
        now = (left == step)[:, None]
        outX, outV = torch.where(now, x, outX), torch.where(now, v, outV)
    return {"X": outX, "V": outV}


def _adjugate(A):
    """(adjugate, determinant) of [n, 3, 3] matrices."""
    c0, c1, c2 = A[:, :, 0], A[:, :, 1], A[:, :, 2]
    adj = torch.stack([torch.linalg.cross(c1, c2), torch.linalg.cross(c2, c0), torch.linalg.cross(c0, c1)], 1)
    return adj, (adj[:, 0] * c0).sum(1)


def _polar(F):
    """Closest proper rotations of [n, 3, 3] matrices: Newton's iteration, an SVD for the flat and inverted ones."""
    flat = _adjugate(F)[1] < 0.1
    R = torch.where(flat[:, None, None], torch.eye(3, dtype=F.dtype, device=F.device), F)
    for _ in range(9):
        adj, det = _adjugate(R)
        R = 0.5 * (R + (adj / det[:, None, None]).transpose(1, 2))
    if bool(flat.any()):
        U, _, Vh = torch.linalg.svd(F[flat])
        U[:, :, 2] *= torch.sign(torch.linalg.det(U) * torch.linalg.det(Vh))[:, None]
        R[flat] = U @ Vh
    return R


def _system(T, BB, mdt2, nv, dev):
    """K = diag(M / h^2) + sum_t c_t B_t^T B_t as a CSR matrix."""
    rows = T[:, :, None].expand(-1, 4, 4).reshape(-1)
    cols = T[:, None, :].expand(-1, 4, 4).reshape(-1)
    d = torch.arange(nv, device=dev)
    at = torch.stack([torch.cat([rows, d]), torch.cat([cols, d])])
    return torch.sparse_coo_tensor(at, torch.cat([BB.reshape(-1), mdt2]), (nv, nv)).coalesce().to_sparse_csr()


def _cg(K, diag, b, x):
    """Jacobi-preconditioned conjugate gradients, the three columns together."""
    r = b - K @ x
    z = r / diag
    p, rz = z, (r * z).sum(0)
    stop = 1e-26 * (b * b / diag).sum(0)
    for it in range(3000):
        if it % 16 == 0 and bool((rz <= stop).all()):
            break
        q = K @ p
        a = torch.where(rz > 0, rz / (p * q).sum(0).clamp_min(1e-300), torch.zeros_like(rz))
        x, r = x + a * p, r - a * q
        z = r / diag
        rn = (r * z).sum(0)
        p = z + torch.where(rz > 0, rn / rz.clamp_min(1e-300), torch.zeros_like(rz)) * p
        rz = rn
    return x
