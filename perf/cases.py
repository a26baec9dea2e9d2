"""The work whose speed this repository is measured by: what a simulation built
on the framework calls in its Newton loop, through the public entry points.

Kinds of case:

* ``contact``: ``ContactPipeline.iteration`` -- the whole contact part of one
  Newton iteration (hierarchy refit, edge-edge and point-triangle detection,
  barrier force and Hessian, the contact matrix, the energy, the CCD step
  bound) -- on two cubes, a bundle of rods in contact, or a screw and its nut;
  with ``host`` the inputs and the force are in pinned host memory
  (``iteration_host``).
* ``system``: ``FEMContactSolver.compute_A`` + ``compute_rhs`` -- the Newton
  matrix and right-hand side of deformable rods wound around one another.
* ``search``: ``FEMContactSolver.line_search`` from a given direction.
* ``solve``: the preconditioned solve of one Newton system, block Jacobi or the
  learned factor (whose build is part of it, as in the Newton loop).
* ``train``: loss and parameter gradients of the learned preconditioner over a
  mini-batch of systems (the backward direction).
* ``mixed``: ``MixedSolver.compute_A`` -- deformable cubes and affine balls in
  one Newton system.
* ``bodies``: ``FixedBVHAffineBodyDynamics.compute_A`` and its CCD bound --
  affine bodies alone.
"""
import functools
import math

import numpy as np
import torch

from ipc_warp_b200 import scenes

H2 = (5e-3) ** 2  # squared time step of the synthetic Newton systems


def listed():
    return [
        # two unit cubes of 8^3 cells (729 vertices each) in contact: the
        # smallest scene in use, bound by launches and latency
        dict(name="cubes", kind="contact", scene="cubes", n=8, gap=5e-4, fp64=False, host=False),
        # nine short rods in the double-precision build, which runs serve as
        # the error oracle of the float one; an odd number of cells
        dict(name="rods-f64", kind="contact", scene="rods", side=3, cells=4, length=37, fp64=True, host=False),
        # the rod-twist bundle in its wound contact state (102,800 vertices,
        # 0.74M contact pairs): an ordinary, contact-heavy scene
        dict(name="rods", kind="contact", scene="rods", side=4, cells=4, length=256, fp64=False, host=False),
        # a part of the screw and nut at an odd number of columns, driven by a
        # program whose positions and directions live in host memory
        dict(name="screw-host", kind="contact", scene="screw", columns=306, turns=5, fp64=False, host=True),
        # the screw and nut of the benchmark (741,120 vertices, 6M CCD
        # candidates): the largest contact scene
        dict(name="screw", kind="contact", scene="screw", columns=640, turns=12, fp64=False, host=False),
        # Newton matrix and right-hand side of the wound rod bundle
        dict(name="system-rods", kind="system", side=4, length=256, theta=0.3, fp64=False),
        # line search on a smaller bundle from a direction that unwinds it
        dict(name="search-rods", kind="search", side=3, length=121, theta=0.13, fp64=False),
        # the solve, with block Jacobi on the bundle of 102,800 vertices ...
        dict(name="solve-jacobi", kind="solve", side=4, length=256, learned=False, fp64=False),
        # ... and with the learned factor on a part of it
        dict(name="solve-learned", kind="solve", side=3, length=200, learned=True, fp64=False),
        # one mini-batch of the preconditioner's training
        dict(name="train", kind="train", side=2, length=64, batch=3),
        # affine balls over settled stacks of deformable cubes on the ground
        dict(name="mixed", kind="mixed", balls=16, cells=4, fp64=False),
        # a pile of affine balls on a slab, per-body hierarchies
        dict(name="bodies", kind="bodies", side=5, layers=2, subdiv=3, fp64=False),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["contact", "contact", "contact", "contact", "system", "search", "solve", "solve", "train",
                       "mixed", "bodies"])
    fp64 = rng.random() < 0.25
    if kind == "contact":
        scene = rng.choice(["cubes", "rods", "screw"])
        host = rng.random() < 0.25
        if scene == "cubes":
            return dict(kind=kind, scene=scene, n=rng.randint(4, 20), gap=rng.choice([2e-4, 3e-4, 5e-4, 7e-4]),
                        fp64=fp64, host=host)
        if scene == "rods":
            return dict(kind=kind, scene=scene, side=rng.randint(2, 4), cells=rng.randint(2, 4), length=log(12, 256),
                        fp64=fp64, host=host)
        # columns - rows a pitch has to be even
        return dict(kind=kind, scene=scene, columns=2 * log(80, 320), turns=rng.randint(2, 12 if not fp64 else 6),
                    fp64=fp64, host=host)
    if kind in ("system", "search"):
        length = log(16, 256)
        return dict(kind=kind, side=rng.randint(2, 4), length=length,
                    theta=round(length * rng.uniform(8e-4, 1.2e-3), 3), fp64=fp64)
    if kind == "solve":
        return dict(kind=kind, side=rng.randint(2, 4), length=log(16, 256), learned=rng.random() < 0.5,
                    fp64=rng.random() < 0.1)
    if kind == "train":
        return dict(kind=kind, side=rng.randint(2, 3), length=log(16, 96), batch=rng.randint(1, 4))
    if kind == "mixed":
        return dict(kind=kind, balls=rng.randint(2, 16), cells=rng.randint(2, 4), fp64=fp64)
    return dict(kind=kind, side=rng.randint(2, 5), layers=rng.randint(1, 3), subdiv=rng.randint(2, 3), fp64=fp64)


# ------------------------------------------------------------------- geometry
# The meshes do not depend on the seed and are kept; every seed moves the
# vertices by its own jitter and has its own direction.
@functools.lru_cache(maxsize=None)
def _cubes(n, gap):
    return scenes.two_cubes(n=n, gap=gap, jitter=0.0)


@functools.lru_cache(maxsize=None)
def _rods(side, cells, length, packed=True):
    return scenes.rod_bundle(n_rods_side=side, cells=(cells, cells, length), gap_over_dhat=0.5 if packed else None,
                             jitter_over_dhat=0.0)


@functools.lru_cache(maxsize=2)
def _screw(columns, turns):
    # a coarser thread needs the clearance that its facets' sagitta takes up
    clearance = 1e-4 * (640 / columns) ** 2
    return scenes.screw_and_nut(n_theta=columns, turns=turns, clearance=clearance, dhat=0.5 * clearance)


def _moved(base, rng, amount):
    """A copy of the scene with every vertex moved by up to ``amount``."""
    x = base.x + rng.uniform(-amount, amount, size=base.x.shape)
    return scenes.Scene(name=base.name, x=x, xcs=x.copy(), edges=base.edges, triangles=base.triangles, body=base.body,
                        tets=base.tets, dhat=base.dhat, kappa=base.kappa, meta=base.meta)


def _contact_scene(case, seed):
    """The scene and a Newton direction dx (the step is x - dx)."""
    rng = np.random.default_rng(seed)
    if case["scene"] == "cubes":
        sc = _moved(_cubes(case["n"], case["gap"]), rng, 1e-5)
        dx = rng.normal(scale=0.2 * sc.dhat, size=sc.x.shape)
        dx[sc.body == 1, 1] += 3.0 * sc.dhat  # the upper cube comes down
        return sc, dx
    if case["scene"] == "rods":
        base = _rods(case["side"], case["cells"], case["length"])
        sc = _moved(base, rng, 0.05 * base.dhat)
        dx = rng.normal(scale=0.3 * sc.dhat, size=sc.x.shape)
        dx[:, :2] += 0.02 * (sc.x[:, :2] - sc.x[:, :2].mean(0)) / sc.meta["width"] * sc.dhat  # the bundle closes
        return sc, dx
    sc = _moved(_screw(case["columns"], case["turns"]), rng, 1e-7)
    return sc, scenes.screw_direction(sc, seed=seed)  # the nut turns at 4 rad/s


def _dtype(case):
    return torch.float64 if case.get("fp64") else torch.float32


def _device():
    return torch.device("cuda")


# -------------------------------------------------------------- Newton systems
@functools.lru_cache(maxsize=None)
def _elastic(side, length):
    """Block pattern and values of h^2 K + springs' slots of a rod bundle:
    linear-elastic tets (E = 1e6, nu = 0.45, rho = 1000), clamped ends, and
    one spring between each pair of facing vertices of neighbouring rods."""
    sc = _rods(side, 4, length)
    x, T = sc.x, sc.tets.astype(np.int64)
    n = x.shape[0]
    E, nu, rho = 1e6, 0.45, 1000.0
    mu, lam = E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))
    D = x[T[:, 1:]] - x[T[:, :1]]  # rows are the edge vectors
    vol = np.abs(np.linalg.det(D)) / 6.0
    G = np.linalg.inv(D)  # columns: gradients of the barycentric coordinates 1..3
    grad = np.concatenate([-G.sum(2)[:, None, :], np.swapaxes(G, 1, 2)], axis=1)  # (t, 4, 3)
    dot = np.einsum("tia,tja->tij", grad, grad)
    outer = np.einsum("tia,tjb->tijab", grad, grad)
    K = lam * outer + mu * np.swapaxes(outer, 3, 4) + mu * dot[..., None, None] * np.eye(3)
    K *= (H2 * vol)[:, None, None, None, None]
    mass = np.bincount(T.ravel(), weights=np.repeat(rho * vol / 4.0, 4), minlength=n)
    z = x[:, 2]
    clamped = (z <= z.min() + 1e-9) | (z >= z.max() - 1e-9)
    # vertex (i, j, k) of rod r is r * nv + (i * 5 + j) * (length + 1) + k
    nv = 25 * (length + 1)
    k = np.arange(length + 1)
    a, b, axis = [], [], []
    for ra in range(side):
        for rb in range(side):
            r = ra * side + rb
            for j in range(5):
                if ra + 1 < side:  # face x = width against face x = 0
                    a.append(r * nv + (20 + j) * (length + 1) + k)
                    b.append((r + side) * nv + j * (length + 1) + k)
                    axis.append(np.zeros_like(k))
                if rb + 1 < side:
                    a.append(r * nv + (j * 5 + 4) * (length + 1) + k)
                    b.append((r + 1) * nv + j * 5 * (length + 1) + k)
                    axis.append(np.ones_like(k))
    a, b, axis = np.concatenate(a), np.concatenate(b), np.concatenate(axis)
    rows = np.concatenate([np.arange(n), np.repeat(T, 4, axis=1).ravel(), a, b])
    cols = np.concatenate([np.arange(n), np.tile(T, (1, 4)).ravel(), b, a])
    key, slot = np.unique(rows * n + cols, return_inverse=True)
    vals = np.zeros((key.size, 9))
    nt = 16 * T.shape[0]
    flat = K.reshape(nt, 9)
    for c in range(9):
        vals[:, c] = np.bincount(slot[n:n + nt], weights=flat[:, c], minlength=key.size)
    offsets = np.searchsorted(key, np.arange(n + 1) * n)
    return dict(n=n, offsets=offsets.astype(np.int32), cols=(key % n).astype(np.int32), vals=vals, diag=slot[:n],
                mass=mass, clamped=clamped, a=a, b=b, axis=axis, ab=slot[n + nt:n + nt + a.size],
                ba=slot[n + nt + a.size:])


def _newton_system(side, length, seed):
    """Offsets, columns and float64 blocks of M + h^2 K + contact springs
    (stiffness over four decades, as barriers give) and a right-hand side;
    rounded to float32, so that every precision starts from the same numbers."""
    e = _elastic(side, length)
    rng = np.random.default_rng(seed)
    vals = e["vals"].copy()
    m = e["mass"] * rng.uniform(0.8, 1.25, e["n"])
    m = m + np.where(e["clamped"], 1e3 * m, 0.0)
    for c in (0, 4, 8):
        vals[e["diag"], c] += m
    s = e["mass"].mean() * 10.0 ** rng.uniform(-1.0, 3.0, e["a"].size)
    c = 4 * e["axis"]
    np.add.at(vals, (e["diag"][e["a"]], c), s)
    np.add.at(vals, (e["diag"][e["b"]], c), s)
    np.add.at(vals, (e["ab"], c), -s)
    np.add.at(vals, (e["ba"], c), -s)
    rhs = e["mass"].mean() * 1e-4 * rng.normal(size=(e["n"], 3))
    return e["offsets"], e["cols"], vals.astype(np.float32), rhs.astype(np.float32)


def _bsr(offsets, cols, vals, dtype):
    from ipc_warp_b200.bsr import BsrMatrix

    n, nnz = offsets.size - 1, cols.size
    A = BsrMatrix(n, n, nnz, dtype, _device())
    A.offsets.copy_(torch.from_numpy(offsets))
    A.columns.copy_(torch.from_numpy(cols))
    A.values.copy_(torch.from_numpy(vals).view(nnz, 3, 3))
    A.nnz_dev.fill_(nnz)
    return A


def _train_seeds(case, seed):
    return [1000 * seed + k for k in range(case["batch"])]


def _most_blocks(case):
    """More blocks than the scene's contact matrix has, and fewer than the
    framework allots for its pairs (16 each)."""
    if case["scene"] == "cubes":
        return 288 * case["n"] ** 2
    if case["scene"] == "rods":
        return 8 * _rod_counts(case["side"], case["cells"], case["length"])[1]
    return 4 * 8 * case["columns"] * 16 * case["turns"]


# --------------------------------------------------------------------- prepare
def _rod_solver(case, seed):
    """FEMContactSolver of StVK rods, packed, wound by theta and jittered, the
    clamped ends one step of the 2 rad/s counter-rotation further."""
    from ipc_warp_b200.newton import FEMContactSolver

    base = _rods(case["side"], 4, case["length"])
    rng = np.random.default_rng(seed)
    fixed, _ = scenes.twist_targets(base, omega=2.0)
    sc = scenes.Scene(name=base.name, x=base.x, xcs=base.x, edges=base.edges, triangles=base.triangles, body=base.body,
                      tets=base.tets, dhat=base.dhat, kappa=1e13, meta=base.meta)
    s = FEMContactSolver(sc, material="stvk", E=1e6, nu=0.45, h=5e-3, fixed=fixed, gravity=(0.0, 0.0, 0.0),
                         dtype=_dtype(case), device=_device(), tol=1e-6, maxiter=20000)
    jitter = rng.uniform(-0.05, 0.05, size=base.x.shape) * base.dhat
    x = scenes.twist_bundle(sc, case["theta"]) + jitter
    target = scenes.twist_bundle(sc, case["theta"] + 2.0 * 5e-3)
    s.states.x.copy_(torch.as_tensor(x))
    s.states.x0.copy_(s.states.x)
    s.x_target.copy_(torch.as_tensor(np.where(fixed[:, None], target, base.x)))
    # a direction that takes a tenth of the winding back (x - dx)
    back = scenes.twist_bundle(sc, 0.9 * case["theta"])
    dx = x - back + rng.normal(scale=0.02 * base.dhat, size=x.shape)
    dx[fixed] = (x - target)[fixed]
    s.states.dx.copy_(torch.as_tensor(dx))
    return s


def prepare(case, seed):
    kind = case["kind"]
    dtype, dev = _dtype(case), _device()
    if kind == "contact":
        from ipc_warp_b200.pipeline import ContactPipeline

        sc, dx = _contact_scene(case, seed)
        pipe = ContactPipeline.from_scene(sc, dtype=dtype, device=dev)
        st = dict(kind=kind, host=case["host"], pipe=pipe, blocks=_most_blocks(case),
                  dx=torch.as_tensor(dx, dtype=dtype, device=dev))
        if case["host"]:
            st["x"] = torch.as_tensor(sc.x, dtype=dtype).pin_memory()
            st["dx"] = torch.as_tensor(dx, dtype=dtype).pin_memory()
            st["b"] = torch.empty_like(st["x"]).pin_memory()
        return st
    if kind in ("system", "search"):
        s = _rod_solver(case, seed)
        v, e, _, _ = _rod_counts(case["side"], 4, case["length"])
        return dict(kind=kind, s=s, x=s.states.x.clone(), blocks=15 * v + 6 * e)
    if kind == "solve":
        from ipc_warp_b200.learned import DEFAULT_WEIGHTS, Net, Pool
        from ipc_warp_b200.newton import DevicePcg

        offsets, cols, vals, rhs = _newton_system(case["side"], case["length"], seed)
        st = dict(kind=kind, A=_bsr(offsets, cols, vals, dtype), b=torch.as_tensor(rhs, dtype=dtype, device=dev),
                  pcg=DevicePcg(), dinv=None, net=None)
        if case["learned"]:
            st["net"], st["pool"] = Net.load(DEFAULT_WEIGHTS, device=dev), Pool()
        return st
    if kind == "train":
        from ipc_warp_b200.learned import DEFAULT_WEIGHTS, Net, System

        net = Net.load(DEFAULT_WEIGHTS, device=dev)
        systems = [System.from_bsr(_bsr(*_newton_system(case["side"], case["length"], k)[:3], torch.float32))
                   for k in _train_seeds(case, seed)]
        return dict(kind=kind, net=net, systems=systems, grad=torch.zeros_like(net.params))
    if kind == "mixed":
        from ipc_warp_b200.bsr import BsrMatrix
        from ipc_warp_b200.mixed import MixedSolver

        sc = scenes.wrecking_balls(n_balls=case["balls"], cube_cells=case["cells"], subdiv=3, ground_quads=100, seed=seed)
        # settled stacks: the facing gaps of 1.5e-3 are inside the barrier
        sc.dhat = 2e-3
        rng = np.random.default_rng(seed)
        sc.fem.x = sc.fem.x + rng.uniform(-0.05, 0.05, size=sc.fem.x.shape) * sc.dhat
        s = MixedSolver(sc, E=5e5, nu=0.4, h=1e-2, dtype=dtype, device=dev, maxiter=2000)
        # a copy of the matrix in arrays of one size (the solver's own grow)
        return dict(kind=kind, s=s, copy=BsrMatrix(s.nq, s.nq, 40 * s.nq + 20000, dtype, dev))
    from ipc_warp_b200.abd import FixedBVHAffineBodyDynamics

    cfg = scenes.abd_balls(n_side=case["side"], layers=case["layers"], subdiv=case["subdiv"], gap=6e-4, drop=6e-4,
                           seed=seed)
    s = FixedBVHAffineBodyDynamics(1e-2, affine_stiffness=1e8, contact_kappa=1e10, dhat=1e-3, dtype=dtype, device=dev,
                                   **cfg)
    rng = np.random.default_rng(seed)
    dq = rng.normal(scale=1e-3, size=tuple(s.abd_states.dx.shape))
    dq[4 * (s.n_bodies - 1):] = 0.0  # the slab is fixed
    s.abd_states.dx.copy_(torch.as_tensor(dq))
    return dict(kind=kind, s=s)


# ------------------------------------------------------------------------- run
def _matrix(A, blocks):
    """The matrix in its first ``blocks`` slots: more than it has blocks, the
    rest zero."""
    return dict(offsets=A.offsets, columns=A.columns[:blocks], values=A.values[:blocks])


def run(state):
    kind = state["kind"]
    if kind == "contact":
        pipe = state["pipe"]
        if state["host"]:
            r = pipe.iteration_host(state["x"], state["dx"], state["b"])
            force = state["b"]
        else:
            r = pipe.iteration(state["dx"])
            force = pipe.b
        return dict(n_ee=r.n_ee, n_pt=r.n_pt, energy=r.energy, alpha=r.alpha, force=force,
                    hessian=_matrix(pipe.collision_hessian, state["blocks"]))
    if kind == "system":
        s = state["s"]
        A = s.compute_A()
        rhs = s.compute_rhs()
        return dict(matrix=_matrix(A, state["blocks"]), rhs=rhs)
    if kind == "search":
        s = state["s"]
        s.states.x.copy_(state["x"])
        alpha = s.line_search()
        return dict(alpha=alpha, x=s.states.x)
    if kind == "solve":
        A = state["A"]
        if state["net"] is None:
            from ipc_warp_b200.newton import JacobiPrecond

            M = JacobiPrecond(A, state["dinv"])
            state["dinv"] = M.dinv
            x, _, _, _ = state["pcg"].solve(A, state["b"], M, 1e-6, 5000)
            return dict(x=x)
        from ipc_warp_b200.learned import LearnedFactor

        M = LearnedFactor(state["net"], A, pool=state["pool"])
        x, _, _, _ = state["pcg"].solve(A, state["b"], M, 1e-6, 5000)
        return dict(x=x, factor=M.G)
    if kind == "train":
        from ipc_warp_b200 import learned as L

        net, grad = state["net"], state["grad"].zero_()
        loss = 0.0
        for sysm in state["systems"]:
            H, tape = L.forward(net, sysm, training=True)
            nz = L.normalize(sysm, H)
            L.backward(net, sysm, tape, L.loss_grad(sysm, nz, weight=1.0 / len(state["systems"])), grad)
            loss += nz.loss / len(state["systems"])
        return dict(loss=loss, grad=grad)
    s = state["s"]
    A = s.compute_A()
    if kind == "mixed":
        B, nnz = state["copy"], A.nnz_sync()
        B.offsets.copy_(A.offsets)
        B.columns[:nnz].copy_(A.columns[:nnz])
        B.values[:nnz].copy_(A.values[:nnz])
        return dict(matrix=_matrix(B, B.columns.shape[0]), rhs=s.compute_rhs())
    alpha = s.line_search_upper_bound()
    nnz = A.nnz_sync()  # the pairs of touching bodies
    return dict(matrix=_matrix(A, nnz), rhs=s.compute_rhs(), alpha=alpha)


# ------------------------------------------------------------------------ work
def _rod_counts(side, cells, length):
    """Vertices, surface edges and triangles, tets of a rod bundle."""
    rods = side * side
    tris = 4 * (2 * cells * cells + 4 * cells * length) // 2
    return (rods * (cells + 1) ** 2 * (length + 1), rods * tris * 3 // 2, rods * tris,
            rods * 5 * cells * cells * length)


def _solve_flops(side, length, iterations):
    v = _rod_counts(side, 4, length)[0]
    return v, 15 * v, 18 * 15 * v * iterations


def work(case):
    """Inputs read once and outputs written once.  The number of contact
    pairs and blocks is the scenes' own (pairs per surface edge and blocks per
    pair as these generators give them)."""
    kind = case["kind"]
    f = 8 if case.get("fp64") else 4
    if kind == "contact":
        if case["scene"] == "cubes":
            n = case["n"]
            v, t = 2 * (n + 1) ** 3, 2 * 12 * n * n
            e, blocks = t * 3 // 2, 3 * n * n
        elif case["scene"] == "rods":
            v, e, t, _ = _rod_counts(case["side"], case["cells"], case["length"])
            share = 1.0 - 1.0 / case["side"]  # of the rods' long sides that face another rod
            blocks = int(5.3 * share * e)
        else:
            v = 6 * case["columns"] * (16 * case["turns"])
            t = 8 * case["columns"] * (16 * case["turns"])
            e, blocks = t * 3 // 2, int(1.2 * t)
        # x, rest positions, dx, bodies, edges, triangles; force, matrix
        bytes_ = v * (3 * 3 * f + 4) + 8 * e + 12 * t + v * 3 * f + blocks * (9 * f + 4) + 4 * v
        return dict(bytes=bytes_, flops=0)
    if kind in ("system", "search"):
        v, e, t, tets = _rod_counts(case["side"], 4, case["length"])
        ins = v * (5 * 3 * f + 4 + 8) + 8 * e + 12 * t + tets * (16 + 10 * f)
        if kind == "search":
            return dict(bytes=2 * ins + v * 3 * f, flops=0)  # the energy at both ends of the step
        return dict(bytes=ins + int(15 * v) * (9 * f + 4) + v * 3 * f, flops=0)
    if kind == "solve":
        # the matrix once; about 180 products with it (80 with the learned factor)
        v, blocks, flops = _solve_flops(case["side"], case["length"], 80 if case["learned"] else 180)
        net = 2 * (4 * (blocks * 64 * 64 + v * 4 * 64 * 64) + blocks * 16 * 64) if case["learned"] else 0
        return dict(bytes=blocks * (9 * f + 4) + v * 6 * f + (36 * blocks if case["learned"] else 0),
                    flops=flops + net)
    if kind == "train":
        v, blocks, _ = _solve_flops(case["side"], case["length"], 0)
        net = 2 * (4 * (blocks * 64 * 64 + v * 4 * 64 * 64) + blocks * 16 * 64)
        return dict(bytes=case["batch"] * blocks * (36 + 2 * 32 + 4 * 128), flops=3 * case["batch"] * net)
    if kind == "mixed":
        n, b = case["cells"], case["balls"]
        cubes = 8 * b
        v, tets = cubes * (n + 1) ** 3, cubes * 5 * n ** 3
        surface = b * 642 + 101 * 101
        t = b * 1280 + 20000 + cubes * 12 * n * n
        blocks = 15 * v + 8 * b * 900
        return dict(bytes=(v + surface) * 3 * 3 * f + 24 * t + tets * (16 + 10 * f) + blocks * (9 * f + 4) + v * 3 * f,
                    flops=0)
    bodies = case["side"] ** 2 * case["layers"]
    t = bodies * 20 * 4 ** case["subdiv"] + 600
    return dict(bytes=(t // 2) * 3 * 3 * f + 24 * t + bodies * bodies * 16 * 9 * f // 4, flops=0)


# ----------------------------------------------------------------------- exact
def _segment_pairs(x, a, b):
    """Closest points of segment pairs (float64): the weights c (n, 4) with
    r = sum_k c_k x_k, the difference of the closest points."""
    p1, q1, p2, q2 = x[a[:, 0]], x[a[:, 1]], x[b[:, 0]], x[b[:, 1]]
    d1, d2, r = q1 - p1, q2 - p2, p1 - p2
    A, B, C = (d1 * d1).sum(1), (d1 * d2).sum(1), (d2 * d2).sum(1)
    D, E = (d1 * r).sum(1), (d2 * r).sum(1)
    den = A * C - B * B
    s = torch.where(den > 0, ((B * E - C * D) / den.clamp_min(1e-300)), torch.zeros_like(den)).clamp(0, 1)
    t = ((B * s + E) / C).clamp(0, 1)
    s = ((B * t - D) / A).clamp(0, 1)
    best = None
    # the interior solution and the four end points against the other segment
    zero, one = torch.zeros_like(s), torch.ones_like(s)
    for u, v in ((s, t), (zero, (E / C).clamp(0, 1)), (one, ((B + E) / C).clamp(0, 1)), ((-D / A).clamp(0, 1), zero),
                 (((B - D) / A).clamp(0, 1), one)):
        c = torch.stack([1 - u, u, v - 1, -v], 1)
        d = (p1 + u[:, None] * d1 - p2 - v[:, None] * d2).square().sum(1)
        if best is None:
            best, w = d, c
        else:
            w = torch.where((d < best)[:, None], c, w)
            best = torch.minimum(d, best)
    return w


def _point_triangles(x, p, t):
    """Weights (n, 4) of the closest-point difference of point-triangle pairs."""
    P, T = x[p], x[t]
    best, w = None, None
    ab, ac, ap = T[:, 1] - T[:, 0], T[:, 2] - T[:, 0], P - T[:, 0]
    a, b, c = (ab * ab).sum(1), (ab * ac).sum(1), (ac * ac).sum(1)
    d, e = (ab * ap).sum(1), (ac * ap).sum(1)
    den = a * c - b * b
    v, u = (c * d - b * e) / den, (a * e - b * d) / den
    inside = (u >= 0) & (v >= 0) & (u + v <= 1)
    face = torch.stack([1 - u - v, v, u], 1)
    options = [torch.where(inside[:, None], face, face.new_tensor([1.0, 0.0, 0.0]))]
    for i, j in ((0, 1), (1, 2), (2, 0)):
        e1 = T[:, j] - T[:, i]
        s = (((P - T[:, i]) * e1).sum(1) / (e1 * e1).sum(1)).clamp(0, 1)
        o = torch.zeros_like(face)
        o[:, i], o[:, j] = 1 - s, s
        options.append(o)
    for o in options:
        dist = (P - (o[:, :, None] * T).sum(1)).square().sum(1)
        if best is None:
            best, w = dist, o
        else:
            w = torch.where((dist < best)[:, None], o, w)
            best = torch.minimum(dist, best)
    return torch.cat([torch.ones_like(best)[:, None], -w], 1)


def _near(lo, hi, lo2, hi2, chunk=1024):
    """Index pairs of overlapping boxes."""
    out = []
    for k in range(0, lo.shape[0], chunk):
        ok = torch.ones(min(chunk, lo.shape[0] - k), lo2.shape[0], dtype=torch.bool, device=lo.device)
        for c in range(3):
            ok &= (lo[k:k + chunk, None, c] <= hi2[None, :, c]) & (hi[k:k + chunk, None, c] >= lo2[None, :, c])
        i, j = ok.nonzero(as_tuple=True)
        out.append(torch.stack([i + k, j], 1))
    return torch.cat(out)


def _contact_exact(case, seed):
    """Energy and force of the barrier in 64 bits, by all pairs of boxes."""
    sc, _ = _contact_scene(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    edges = torch.as_tensor(sc.edges.reshape(-1, 2).astype(np.int64), device=dev)
    tris = torch.as_tensor(sc.triangles.reshape(-1, 3).astype(np.int64), device=dev)
    if edges.shape[0] > 40000:
        return None
    x = torch.as_tensor(sc.x, dtype=_dtype(case), device=dev).double().requires_grad_(True)
    rest = x.detach()
    dhat = sc.dhat
    with torch.no_grad():
        eb = x[edges]
        lo, hi = eb.amin(1), eb.amax(1)
        pairs = _near(lo - dhat, hi + dhat, lo, hi)
        pairs = pairs[pairs[:, 0] < pairs[:, 1]]
        a, b = edges[pairs[:, 0]], edges[pairs[:, 1]]
        apart = (a[:, :, None] != b[:, None, :]).all(2).all(1)
        a, b = a[apart], b[apart]
        w = _segment_pairs(x, a, b)
        ids = torch.cat([a, b], 1)
        d = (w[:, :, None] * x[ids]).sum(1).norm(dim=1)
        keep = d < dhat
        ids, w = ids[keep], w[keep]
        tb = x[tris]
        pt = _near(x - dhat, x + dhat, tb.amin(1), tb.amax(1))
        tri = tris[pt[:, 1]]
        pt, tri = pt[(tri != pt[:, :1]).all(1)], tri[(tri != pt[:, :1]).all(1)]
        wp = _point_triangles(x, pt[:, 0], tri)
        pids = torch.cat([pt[:, :1], tri], 1)
        d = (wp[:, :, None] * x[pids]).sum(1).norm(dim=1)
        pids, wp = pids[d < dhat], wp[d < dhat]

    def barrier(i, c):
        d2 = (c[:, :, None] * x[i]).sum(1).square().sum(1)
        h2 = dhat * dhat
        return -sc.kappa * (d2 - h2) ** 2 * torch.log(d2 / h2)

    X = x[ids]
    cross = torch.linalg.cross(X[:, 1] - X[:, 0], X[:, 3] - X[:, 2]).square().sum(1)
    R = rest[ids]
    eps = 1e-3 * (R[:, 1] - R[:, 0]).square().sum(1) * (R[:, 3] - R[:, 2]).square().sum(1)
    ratio = cross / eps
    mollifier = torch.where(ratio < 1, (2 - ratio) * ratio, torch.ones_like(ratio))
    e = (mollifier * barrier(ids, w)).sum() + barrier(pids, wp).sum()
    e.backward()
    # the projected Hessian's blocks, the pair counts and the step bound are
    # compared with what the same inputs gave before
    return dict(n_ee=None, n_pt=None, energy=float(e.detach()) * 1e-4, alpha=None, force=-x.grad, hessian=None)


def _net_exact(side, length, seed, params):
    """(loss, G) of the learned factor in 64 bits: the message-passing net on
    the scaled blocks, the row directions and their exact normalisation."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    offsets, cols, vals, _ = _newton_system(side, length, seed)
    off = torch.as_tensor(offsets.astype(np.int64), device=dev)
    col = torch.as_tensor(cols.astype(np.int64), device=dev)
    V = torch.as_tensor(vals, device=dev).double().view(-1, 3, 3)
    n = off.numel() - 1
    deg = (off[1:] - off[:-1])
    row = torch.repeat_interleave(torch.arange(n, device=dev), deg)
    diag = (row == col).nonzero().view(-1)
    s = V[diag].diagonal(dim1=1, dim2=2).rsqrt()
    A = V * s[row][:, :, None] * s[col][:, None, :]
    fro = A.square().sum((1, 2)).sqrt()
    c = torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, row, torch.where(row != col, fro, 0.0 * fro))
    X = torch.zeros(n, 16, dtype=torch.float64, device=dev)
    X[:, :9], X[:, 9], X[:, 10] = A[diag].reshape(n, 9), torch.log1p(deg.double()), c
    Y = torch.zeros(col.numel(), 16, dtype=torch.float64, device=dev)
    Y[:, :9], Y[:, 9], Y[:, 10] = A.reshape(-1, 9), fro, (row == col).double()
    at = 0

    def take(*shape):
        nonlocal at
        k = math.prod(shape)
        at += k
        return params[at - k:at].view(*shape)

    h = torch.relu(X @ take(16, 64) + take(64))
    e = torch.relu(Y @ take(16, 64) + take(64))
    for _ in range(4):
        W1, b1, W2, b2 = take(192, 64), take(64), take(128, 64), take(64)
        m = torch.relu((h @ W1[:64])[row] + (h @ W1[64:128])[col] + e @ W1[128:] + b1)
        mean = torch.zeros_like(h).index_add(0, row, m) / deg[:, None]
        h = h + torch.relu(torch.cat([h, mean], 1) @ W2 + b2)
        e = e + m
    low = (col <= row).nonzero().view(-1)
    out = (e[low] @ take(64, 9) + take(9)).view(-1, 3, 3)
    eye = torch.eye(3, dtype=torch.float64, device=dev)
    rho = (c / (1 + c))[row[low]][:, None, None]
    on = (row[low] == col[low])[:, None, None]
    Hd = torch.where(on, eye, (rho * out - eye) @ A[low])
    # T_ij = sum_k H_ik A_kj over the lower pattern of row i
    li, lk = row[low], col[low]
    key = li * n + lk
    T = torch.zeros_like(Hd)
    for lo in range(0, low.numel(), 1 << 18):
        hi = min(lo + (1 << 18), low.numel())
        cnt = deg[lk[lo:hi]]
        src = torch.repeat_interleave(torch.arange(lo, hi, device=dev), cnt)
        first = torch.repeat_interleave(off[lk[lo:hi]] - torch.cumsum(cnt, 0) + cnt, cnt)
        slot = first + torch.arange(src.numel(), device=dev)
        want = li[src] * n + col[slot]
        pos = torch.searchsorted(key, want).clamp_max(key.numel() - 1)
        ok = key[pos] == want
        T = T.index_add(0, pos[ok], Hd[src[ok]] @ A[slot[ok]])
    M = torch.zeros(n, 3, 3, dtype=torch.float64, device=dev).index_add(0, li, T @ Hd.transpose(1, 2))
    M = 0.5 * (M + M.transpose(1, 2))
    C = torch.linalg.cholesky(M)
    loss = 2.0 * C.diagonal(dim1=1, dim2=2).log().sum() / (3 * n)
    with torch.no_grad():
        G = torch.zeros(col.numel(), 3, 3, dtype=torch.float64, device=dev)
        G[low] = torch.linalg.solve_triangular(C, eye.expand(n, 3, 3), upper=False)[li] @ Hd
    return loss, G


def _params(dev):
    from ipc_warp_b200.learned import DEFAULT_WEIGHTS

    return torch.as_tensor(np.load(DEFAULT_WEIGHTS).astype(np.float64), device=dev)


def _solution(side, length, seed):
    """Block-Jacobi conjugate gradients in 64 bits to 1e-13."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    offsets, cols, vals, rhs = _newton_system(side, length, seed)
    n = offsets.size - 1
    row = np.repeat(np.arange(n), np.diff(offsets))
    A = torch.as_tensor(vals, device=dev).double().view(-1, 3, 3)
    r3 = torch.as_tensor(row, device=dev)
    c3 = torch.as_tensor(cols.astype(np.int64), device=dev)
    Dinv = torch.linalg.inv(A[(r3 == c3).nonzero().view(-1)])
    k = torch.arange(3, device=dev)
    ij = torch.stack([(3 * r3[:, None, None] + k[:, None]).expand(-1, 3, 3).reshape(-1),
                      (3 * c3[:, None, None] + k[None, :]).expand(-1, 3, 3).reshape(-1)])
    S = torch.sparse_coo_tensor(ij, A.reshape(-1), (3 * n, 3 * n)).coalesce().to_sparse_csr()
    b = torch.as_tensor(rhs, device=dev).double()

    def prec(v):
        return torch.bmm(Dinv, v[:, :, None]).squeeze(2)

    x, r = torch.zeros_like(b), b.clone()
    z = prec(r)
    p, rz = z.clone(), (r * z).sum()
    stop = 1e-26 * (b * b).sum()
    for it in range(4000):
        q = (S @ p.reshape(-1, 1)).view(n, 3)
        a = rz / (p * q).sum()
        x = x + a * p
        r = r - a * q
        if it % 16 == 0 and (r * r).sum() <= stop:
            break
        z = prec(r)
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "contact":
        return _contact_exact(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "solve":
        out = dict(x=_solution(case["side"], case["length"], seed))
        if case["learned"]:
            with torch.no_grad():
                out["factor"] = _net_exact(case["side"], case["length"], seed, _params(dev))[1]
        return out
    if kind == "train":
        params = _params(dev).requires_grad_(True)
        total = 0.0
        for k in _train_seeds(case, seed):
            loss, _ = _net_exact(case["side"], case["length"], k, params)
            (loss / case["batch"]).backward()
            total += float(loss.detach()) / case["batch"]
        return dict(loss=total, grad=params.grad)
    # whole Newton systems and searches: no restatement in a few lines
    return None
