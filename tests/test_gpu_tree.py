"""The packed tree the queries walk (csrc/tree.cuh): candidate sets and TOI
against the oracle at sizes around its block, group and level edges (32, 1024
and 32768 leaves), for the discrete query, the CCD query with and without a
contact list to start from, and both in one walk (gpu)."""
import numpy as np
import pytest
import torch

from helpers import sort_records
from ipc_warp_b200.pipeline import ContactPipeline
from ipc_warp_b200.scenes import Scene
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def loose_triangles(n, seed, dhat=0.02):
    """n separate triangles (3n edges, 3n vertices) in a box that keeps a few
    neighbours per triangle; a third of them far away, so that blocks of the
    Morton order span the gap."""
    rng = np.random.default_rng(seed)
    side = max(0.35, 0.22 * n ** (1 / 3))
    c = rng.uniform(0, side, size=(n, 1, 3))
    c[: n // 3] += 40.0 * side
    x = (c + rng.uniform(-0.1, 0.1, size=(n, 3, 3))).reshape(-1, 3)
    t = np.arange(3 * n).reshape(n, 3)
    edges = np.concatenate([t[:, [0, 1]], t[:, [1, 2]], t[:, [0, 2]]])
    return Scene(name="loose", x=x, xcs=x.copy(), edges=edges.astype(np.int32).ravel(),
                 triangles=t.astype(np.int32).ravel(), body=np.repeat(np.arange(n) % 3, 3).astype(np.int32),
                 tets=np.zeros((0, 4), np.int32), dhat=dhat, kappa=1.0)


@pytest.mark.parametrize("n", [1, 10, 11, 341, 342, 10922, 10923])
@pytest.mark.parametrize("fp64", [False, True])
def test_tree_queries_match_oracle(cuda, n, fp64):
    sc = loose_triangles(n, seed=n)
    dtype = torch.float64 if fp64 else torch.float32
    excl = n % 2 == 0
    pipe = ContactPipeline.from_scene(sc, dtype=dtype, device=cuda, exclude_same_body=excl)
    rng = np.random.default_rng(n + 1)
    dx = torch.tensor(rng.normal(scale=0.01, size=sc.x.shape), dtype=dtype, device=cuda)
    x0 = pipe.soup.x_transformed.cpu().numpy()
    x32 = x0.astype(np.float32)
    th = np.float32(sc.thickness)
    kw = dict(exclude_same_body=excl)
    ee = sort_records(po.dcd_ee(x32, sc.edges, sc.body, th, **kw))
    pt = sort_records(po.dcd_pt(x32, sc.triangles, sc.body, th, **kw))
    x1 = (x0 - dx.cpu().numpy())
    toi, st = po.scene_toi(x0, x1, sc.edges, sc.triangles, sc.body, fp64=fp64, **kw)
    assert st == 0
    if n >= 341:
        assert len(ee) and len(pt) and toi < 1.0

    def check(bound):
        assert np.array_equal(sort_records(pipe.contacts_new.records(pipe.n_contacts).cpu().numpy()), ee)
        assert np.array_equal(sort_records(pipe.contacts_pt.records(pipe.n_contacts_pt).cpu().numpy()), pt)
        got = float(pipe.ccd_toi.item())
        assert got <= toi and toi - got <= 1e-6
        assert bound == (0.9 * got if got < 1.0 else 1.0)
        return got

    alone = None
    bound = pipe.collision_free_step(dx)  # no contact list yet
    pipe.detect_collision()
    alone = check(bound)
    assert check(pipe.collision_free_step(dx)) == alone  # started from the list
    for _ in range(2):  # eager, then the replayed graph: one walk for both queries
        r = pipe.iteration(dx)
        assert r.status == 0 and (r.n_ee, r.n_pt) == (len(ee), len(pt))
        assert check(r.alpha) == alone
    pipe.iteration(-dx)  # the lists now belong to the same positions, another direction
    assert check(pipe.collision_free_step(dx)) == alone
    # the lists may be of other positions: only their pairs are tried
    x = pipe.soup.x_transformed.clone()
    pipe.soup.x_transformed.add_(torch.tensor(rng.normal(scale=0.05, size=sc.x.shape), dtype=dtype, device=cuda))
    pipe.detect_collision()
    pipe.soup.x_transformed.copy_(x)
    assert pipe.collision_free_step(dx) == bound


def test_both_queries_with_a_small_staging_list(cuda):
    """Pairs that do not fit the staging list send the staged CCD to the pass
    that solves in place; the discrete records are not affected."""
    from ipc_warp_b200 import _native as N

    sc = loose_triangles(342, seed=5)
    pipe = ContactPipeline.from_scene(sc, dtype=torch.float32, device=cuda)
    pipe.use_graph = False
    rng = np.random.default_rng(6)
    dx = torch.tensor(rng.normal(scale=0.01, size=sc.x.shape), dtype=torch.float32, device=cuda)
    full = pipe.iteration(dx)
    for cap in (16, 0):
        pipe._toi_ws = torch.empty(N.size("ipcb_toi_workspace", cap), dtype=torch.uint8, device=cuda)
        pipe._toi_ws_pt = torch.empty_like(pipe._toi_ws)
        small = pipe.iteration(dx)
        assert (small.n_ee, small.n_pt, small.alpha, small.status) == (full.n_ee, full.n_pt, full.alpha, 0)


@pytest.mark.parametrize("n", [40, 342, 4700, 9400, 18000])
def test_point_walk_from_any_stored_toi(cuda, n):
    """The point walks form their boxes up to the TOI stored when a warp
    starts; with 16, 16, 8, 4 and 2 warps a query block the records and the
    minimum are the oracle's from whatever word they start."""
    sc = loose_triangles(n, seed=n)
    pipe = ContactPipeline.from_scene(sc, dtype=torch.float32, device=cuda)
    rng = np.random.default_rng(n)
    dx = torch.tensor(rng.normal(scale=0.02, size=sc.x.shape), dtype=torch.float32, device=cuda)
    x0 = pipe.soup.x_transformed.cpu().numpy()
    pt = sort_records(po.dcd_pt(x0, sc.triangles, sc.body, np.float32(sc.thickness)))
    toi, _ = po.scene_toi(x0, x0 - dx.cpu().numpy(), np.zeros(0, np.int32), sc.triangles, sc.body)
    pipe.collision_free_step(dx)  # ccd_x1

    def check(start, found):
        got = float(pipe.ccd_toi.item())
        assert got <= min(start, toi) and min(start, toi) - got <= 1e-6
        if found is not None:
            assert len(found) == len(pt) and np.array_equal(sort_records(found), pt)

    for start in (1.0, 0.6, 0.5 * (toi + 1.0), toi, 0.5 * toi, 0.0):
        start = float(np.float32(start))
        pipe.ccd_toi.fill_(start)
        pipe.contacts_pt.cnt.zero_()
        pipe._both_queries("pt", pipe._toi_ws_pt)
        found = pipe.contacts_pt.records(int(pipe.contacts_pt.cnt.item())).cpu().numpy()
        pipe._solve_staged("pt", pipe._toi_ws_pt)
        check(start, found)
        pipe.ccd_toi.fill_(start)
        pipe._ccd_query("pt", 0, pipe.soup.n_verts, pipe._toi_ws_pt)
        check(start, None)


@pytest.mark.parametrize("far", [1e17, 3e19, 1e30])
def test_step_far_beyond_the_scene(cuda, far):
    """A diverged direction: boxes whose areas exceed float32."""
    sc = loose_triangles(342, seed=7)
    pipe = ContactPipeline.from_scene(sc, dtype=torch.float32, device=cuda)
    rng = np.random.default_rng(8)
    dx = rng.normal(scale=0.001, size=sc.x.shape).astype(np.float32)
    dx[[5, 600]] = far * rng.normal(size=(2, 3))
    x0 = pipe.soup.x_transformed.cpu().numpy()
    toi, _ = po.scene_toi(x0, x0 - dx, sc.edges, sc.triangles, sc.body)
    dev = torch.tensor(dx, device=cuda)
    for bound in (pipe.collision_free_step(dev), pipe.iteration(dev).alpha):
        got = float(pipe.ccd_toi.item())
        assert got <= toi and toi - got <= 1e-6 and bound == (0.9 * got if got < 1.0 else 1.0)


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("cap", [1 << 16, 40, 0])
def test_toi_of_given_boxes_equals_the_step(cuda, fp64, cap):
    """The CCD queries on boxes the caller formed (whole, and in ranges off the
    32-query blocks; a staging list that fits, overflows, or is none) give the
    TOI of the queries that form their own, also where the caller's triangle
    boxes are wider than the points'."""
    import ctypes

    from ipc_warp_b200 import _native as N

    sc = loose_triangles(342, seed=9)
    dtype = torch.float64 if fp64 else torch.float32
    pipe = ContactPipeline.from_scene(sc, dtype=dtype, device=cuda)
    dx = torch.tensor(np.random.default_rng(10).normal(scale=0.02, size=sc.x.shape), dtype=dtype, device=cuda)
    pipe.collision_free_step(dx)  # ccd_x1
    soup, x1, toi, st = ctypes.byref(pipe.soup.c_struct()), N.ptr(pipe.ccd_x1), pipe.ccd_toi, pipe._status
    ws = torch.empty(N.size("ipcb_toi_workspace", cap), dtype=torch.uint8, device=cuda)

    def value(calls):
        toi.fill_(1.0)
        st.zero_()
        for c in calls:
            c()
        assert int(st.item()) == 0
        return float(toi.item())

    s = N.stream_handle()
    tail = (N.ptr(toi), N.ptr(st), N.ptr(ws), ws.numel(), s)
    cuts = {"ee": (0, 7, 33, 500, pipe.soup.n_edges), "pt": (0, 31, 64, 333, pipe.soup.n_verts)}
    for which, step in (("ee", pipe._toi_ws), ("pt", pipe._toi_ws_pt)):
        n = cuts[which][-1]
        ref = value([lambda: pipe._ccd_query(which, 0, n, step)])
        assert ref < 1.0
        assert value([lambda a=a, b=b: pipe._ccd_query(which, a, b - a, ws)
                      for a, b in zip(cuts[which], cuts[which][1:])]) == ref
        for pad in (1e-7, 0.03):
            if which == "ee":
                lo, hi, bvh = pipe.ccd_edge_lower, pipe.ccd_edge_upper, pipe.ccd_edge_bvh
                N.call("ipcb_swept_edge_aabbs", soup, x1, pad, N.ptr(lo), N.ptr(hi), s)
                bvh.refit(lo, hi)
                head = (soup, x1, ctypes.byref(bvh.c), N.ptr(lo), N.ptr(hi), 0)
                name = "ipcb_edge_edge_toi"
            else:
                lo, hi, bvh = pipe.ccd_triangle_lower, pipe.ccd_triangle_upper, pipe.ccd_triangle_bvh
                N.call("ipcb_swept_triangle_aabbs", soup, x1, pad, N.ptr(lo), N.ptr(hi), s)
                bvh.refit(lo, hi)
                head = (soup, x1, ctypes.byref(bvh.c), 1e-7, 0)
                name = "ipcb_point_triangle_toi"
            assert value([lambda: N.call(name, *head, *tail)]) == ref
            assert value([lambda a=a, b=b: N.call(name + "_range", *head, a, b - a, *tail)
                          for a, b in zip(cuts[which], cuts[which][1:])]) == ref


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("offset", [0.0, 30.0, 1000.0])
def test_touch_bound_keeps_the_minimum_far_from_the_origin(cuda, fp64, offset):
    """The pairs are bounded in float before the double solve; the margin
    covers the rounding of positions far from the origin (the oracle solves
    every pair whose boxes meet)."""
    sc = loose_triangles(200, seed=11)
    sc.x = sc.x + offset * np.array([1.0, -0.7, 0.4])
    dtype = torch.float64 if fp64 else torch.float32
    pipe = ContactPipeline.from_scene(sc, dtype=dtype, device=cuda)
    for seed, scale in ((1, 0.01), (2, 0.1), (3, 1.0)):
        dx = torch.tensor(np.random.default_rng(seed).normal(scale=scale, size=sc.x.shape), dtype=dtype, device=cuda)
        x0 = pipe.soup.x_transformed.cpu().numpy()
        toi, _ = po.scene_toi(x0, x0 - dx.cpu().numpy(), sc.edges, sc.triangles, sc.body, fp64=fp64)
        for run in (pipe.collision_free_step, pipe.iteration):
            run(dx)
            got = float(pipe.ccd_toi.item())
            assert got <= toi and toi - got <= 1e-6


def test_solving_a_staged_list_twice(cuda):
    """The second call of a solve stays inside the list and finds nothing new."""
    from ipc_warp_b200 import _native as N

    sc = loose_triangles(342, seed=12)
    pipe = ContactPipeline.from_scene(sc, dtype=torch.float32, device=cuda)
    dx = torch.tensor(np.random.default_rng(13).normal(scale=0.02, size=sc.x.shape), dtype=torch.float32, device=cuda)
    bound = pipe.collision_free_step(dx)
    for which in ("ee", "pt"):
        pipe.ccd_toi.fill_(1.0)
        pipe._both_queries(which, pipe._toi_ws)
        n = int(pipe._toi_ws[:4].view(torch.int32))  # a list that just holds them
        ws = torch.empty(N.size("ipcb_toi_workspace", n) + 4096, dtype=torch.uint8, device=cuda)
        guard = ws[-4096:]
        guard.fill_(0x5A)
        ws = ws[:-4096]
        pipe._both_queries(which, ws)
        assert int(ws[:4].view(torch.int32)) == n > 0
        pipe._solve_staged(which, ws)
        toi = float(pipe.ccd_toi.item())
        pipe._solve_staged(which, ws)
        assert float(pipe.ccd_toi.item()) == toi and bool((guard == 0x5A).all())
        assert bound <= (0.9 * toi if toi < 1.0 else 1.0)
