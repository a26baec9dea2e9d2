"""Drop-in contact solver base: the Python surface of contact.py (reference
contact.py:444-750) backed by the sm_100a kernels of libipcb200.

A class that mixes in :class:`ContactSolverBase` sets ``self.soup`` (a
:class:`Soup`) before calling ``ContactSolverBase.__init__(self)``, exactly as
with the reference mixin.  Afterwards it has the reference attributes
``bvh_edges``, ``tri_mesh``, ``ccd_edge_bvh``, ``ccd_triangle_bvh``,
``ccd_toi``, ``ccd_x1``, ``contacts_new``, ``contacts_pt``, ``n_contacts``,
``n_contacts_pt``, ``disable_self_collision`` and the methods
``detect_collision()``, ``collision_free_step(dx)``, ``update_bvh()``,
``compute_edge_aabbs()``, ``compute_V()`` and ``_grow_contact_list()``.

Module globals mirror contact.py:14-22 (``_thickness``, ``buffer``,
``contact_volume``, ``disable_self_collision``, ``verbose``); they are read
at call time, so a scene sets ``contact._thickness = dhat / 2`` as with the
reference (dhat = l0 = 2 * _thickness, contact.py:180).
"""
from __future__ import annotations

import ctypes
import warnings
from contextlib import contextmanager, nullcontext
from dataclasses import dataclass
from functools import partial

import torch

from . import _native as N
from . import scalar_types as st
from .lbvh import Bvh

_thickness = 0.01
contact_volume = 10000
buffer = _thickness
eps = 1e-6
disable_self_collision = False
verbose = False

# IPCB_STATUS_STACK | IPCB_STATUS_ROOT_ITERS: a query that ran out of its
# traversal stack, its visit bound or its root iterations may have missed an
# impact, so its TOI is no bound
QUERY_FAILED = 1 | 2


@dataclass
class Soup:
    """fem/geometry.py:165-171.  Positions are (V, 3) tensors of the scalar
    type, index arrays flat int32 like the reference."""
    xcs: torch.Tensor
    triangles: torch.Tensor
    edges: torch.Tensor
    body: torch.Tensor
    x_transformed: torch.Tensor

    @property
    def n_verts(self) -> int:
        return self.xcs.shape[0]

    @property
    def n_edges(self) -> int:
        return self.edges.shape[0] // 2

    @property
    def n_tris(self) -> int:
        return self.triangles.shape[0] // 3

    def c_struct(self, x: torch.Tensor | None = None) -> N.Soup:
        x = self.x_transformed if x is None else x
        if x.dtype not in (torch.float32, torch.float64) or not x.is_contiguous():
            raise ValueError("positions must be contiguous float32/float64 (V, 3)")
        if self.xcs.dtype != x.dtype:
            raise ValueError("xcs and x_transformed must share the scalar type")
        return N.Soup(self.n_verts, self.n_edges, self.n_tris, int(x.dtype == torch.float64), N.ptr(x),
                      N.ptr(self.xcs), N.ptr(self.edges), N.ptr(self.triangles), N.ptr(self.body))

    @staticmethod
    def from_numpy(x, edges, triangles, body, xcs=None, device="cuda", dtype=None) -> "Soup":
        dtype = dtype or st.scalar()
        xt = torch.as_tensor(x, dtype=dtype, device=device).contiguous()
        xr = xt.clone() if xcs is None else torch.as_tensor(xcs, dtype=dtype, device=device).contiguous()
        i32 = lambda a: torch.as_tensor(a, dtype=torch.int32, device=device).reshape(-1).contiguous()
        return Soup(xcs=xr, triangles=i32(triangles), edges=i32(edges), body=i32(body), x_transformed=xt)


class Contacts:
    """contact.py:61-80 ``Contacts`` with its ``XConstraint`` records stored
    as columns: ``a1a2b1b2`` int32 (cap, 4), ``e0e1`` int32 (cap, 2), ``l0``,
    ``alpha``, ``lam`` scalar (cap,), ``cnt`` int32 (1,).  ``htable`` is
    allocated for attribute compatibility; the reference writes it without
    ever reading it (contact.py:183), so it is left at -1."""

    def __init__(self, capacity: int, dtype: torch.dtype, device):
        self.capacity = int(capacity)
        self.dtype = dtype
        self.device = device
        self.a1a2b1b2 = torch.zeros((self.capacity, 4), dtype=torch.int32, device=device)
        self.e0e1 = torch.zeros((self.capacity, 2), dtype=torch.int32, device=device)
        self.l0 = torch.zeros(self.capacity, dtype=dtype, device=device)
        self.alpha = torch.zeros(self.capacity, dtype=dtype, device=device)
        self.lam = torch.zeros(self.capacity, dtype=dtype, device=device)
        self.cnt = torch.zeros(1, dtype=torch.int32, device=device)
        self.htable = torch.full((8191,), -1, dtype=torch.int32, device=device)

    @property
    def list(self) -> "Contacts":
        return self

    def c_struct(self) -> N.Contacts:
        return N.Contacts(N.ptr(self.a1a2b1b2), N.ptr(self.e0e1), N.ptr(self.l0), N.ptr(self.alpha),
                          N.ptr(self.lam), N.ptr(self.cnt), self.capacity)

    def __setattr__(self, name, value):
        object.__setattr__(self, name, value)
        self.__dict__["_addresses"] = None  # of the columns as they were

    def addresses(self) -> tuple:
        """What a captured sequence holds of the list (part of its key)."""
        if self._addresses is None:
            self.__dict__["_addresses"] = (self.capacity, *(c.data_ptr() for c in (
                self.a1a2b1b2, self.e0e1, self.l0, self.alpha, self.lam, self.cnt)))
        return self._addresses

    def grow(self, capacity: int) -> None:
        self.__init__(capacity, self.dtype, self.device)

    def records(self, n: int) -> torch.Tensor:
        """(n, 6) int32 [a1, a2, b1, b2, e0, e1] of the first n records."""
        return torch.cat([self.a1a2b1b2[:n], self.e0e1[:n]], dim=1)


def _edge_aabbs(soup: Soup, x4, pad: float, lower, upper):
    N.call("ipcb_edge_aabbs", ctypes.byref(soup.c_struct()), N.ptr(x4), pad, N.ptr(lower), N.ptr(upper),
           N.stream_handle())


def _triangle_aabbs(soup: Soup, x4, lower, upper):
    N.call("ipcb_triangle_aabbs", ctypes.byref(soup.c_struct()), N.ptr(x4), 0.0, N.ptr(lower), N.ptr(upper),
           N.stream_handle())


def _next_pow2(n: int) -> int:
    return 1 << (max(n, 1) - 1).bit_length()


class ContactSolverBase:
    """contact.py:444-750 mixin.  Requires ``self.soup``."""

    def __init__(self):
        soup: Soup = self.soup
        self.disable_self_collision = disable_self_collision
        dev = soup.xcs.device
        self.device = dev
        dtype = soup.xcs.dtype
        n_edges, n_nodes, n_tris = soup.n_edges, soup.n_verts, soup.n_tris
        f32 = dict(dtype=torch.float32, device=dev)
        self.x4 = torch.zeros((n_nodes, 4), **f32)  # float32 mesh copy (contact.py:476, x_mesh)
        self.bvh_edges = None
        self._edge_boxes = torch.zeros((n_edges, 3), **f32), torch.zeros((n_edges, 3), **f32)
        self.compute_edge_aabbs()
        self.bvh_edges = Bvh(*self._edge_boxes)
        # CCD boxes are refit into the DCD hierarchies (same primitives, same
        # topology); detect_collision refits them back before every query.
        self.ccd_edge_lower = torch.zeros((n_edges, 3), **f32)
        self.ccd_edge_upper = torch.zeros((n_edges, 3), **f32)
        self.ccd_edge_bvh = self.bvh_edges
        self.ccd_toi = torch.ones(1, dtype=dtype, device=dev)
        self.ccd_x1 = torch.zeros_like(soup.x_transformed)
        self.has_triangles = n_tris > 0
        if self.has_triangles:
            self.tri_mesh = None
            self._tri_boxes = torch.zeros((n_tris, 3), **f32), torch.zeros((n_tris, 3), **f32)
            self._triangle_aabbs()
            self.tri_mesh = Bvh(*self._tri_boxes)
            self.ccd_triangle_lower = torch.zeros((n_tris, 3), **f32)
            self.ccd_triangle_upper = torch.zeros((n_tris, 3), **f32)
            self.ccd_triangle_bvh = self.tri_mesh
            # visiting order of the point queries: a warp's 32 vertices are
            # neighbours on the Morton curve (built once, like the hierarchies)
            points = self.x4[:, :3].contiguous()
            self._point_order = Bvh(points, points).sorted.clone()
        self.contacts_new = Contacts(contact_volume, dtype, dev)
        self.contacts_pt = Contacts(contact_volume, dtype, dev)
        self.contacts_list_new = self.contacts_new
        self.contacts_list_pt = self.contacts_pt
        self.n_contacts = 0
        self.n_contacts_pt = 0
        self._status = torch.zeros(1, dtype=torch.int32, device=dev)
        self.query_status = 0  # status word of the last detect_collision / collision_free_step
        self.ccd_refusals = 0  # collision_free_step calls refused for a failed query
        # CCD candidate staging (a query that overflows it is redone inline)
        cap = max(1 << 20, 4 * max(n_edges, n_nodes))
        self._toi_ws = torch.empty(N.size("ipcb_toi_workspace", cap), dtype=torch.uint8, device=dev)
        # both counts and the status; then the TOI (two words) and the status
        self._counts_host = torch.zeros(6, dtype=torch.int32).pin_memory() if dev.type == "cuda" else None

    # ------------------------------------------------------------- branches
    @contextmanager
    def _branch(self, k: int):
        """Launches on side stream k, after what the current stream has
        queued; _join(k) makes the current stream wait for them.  Works inside
        stream capture (the branches become parallel paths of the graph)."""
        streams = self.__dict__.setdefault("_branches", {})
        if k not in streams:
            streams[k] = torch.cuda.Stream(device=self.device)
        streams[k].wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(streams[k]):
            yield streams[k]

    def _join(self, *ks: int):
        for k in ks:
            torch.cuda.current_stream().wait_stream(self._branches[k])

    def _captured(self) -> tuple:
        """What a captured sequence holds by value, or by an address a caller
        may replace: part of the key of every graph, so that all of a
        solver's graphs follow a change at the same call."""
        return (_thickness, buffer, bool(self.disable_self_collision), float(self.contact_stiffness), float(self.h),
                getattr(self, "bvh_rebuild_interval", 0), self.soup.x_transformed.data_ptr(), self.soup.xcs.data_ptr(),
                self.contacts_new.addresses(), self.contacts_pt.addresses())

    # --------------------------------------------------------------- hooks
    def profile_timer(self, name):
        return nullcontext()

    def compute_V(self, ret=True):
        return None

    # --------------------------------------------------------------- boxes
    def _pack(self):
        N.call("ipcb_pack_positions", ctypes.byref(self.soup.c_struct()), N.ptr(self.x4), N.stream_handle())

    def compute_edge_aabbs(self):
        """contact.py:679-681: edge boxes padded by _thickness + buffer."""
        self._pack()
        boxes = self._edge_boxes if self.bvh_edges is None else self.bvh_edges.rewrite()
        _edge_aabbs(self.soup, self.x4, float(_thickness + buffer), *boxes)

    def _triangle_aabbs(self):
        _triangle_aabbs(self.soup, self.x4, *(self._tri_boxes if self.tri_mesh is None else self.tri_mesh.rewrite()))

    @property
    def bvh_edges_lower(self) -> torch.Tensor:
        return self.bvh_edges.lower

    @property
    def bvh_edges_upper(self) -> torch.Tensor:
        return self.bvh_edges.upper

    @property
    def tri_lower(self) -> torch.Tensor:
        return self.tri_mesh.lower

    @property
    def tri_upper(self) -> torch.Tensor:
        return self.tri_mesh.upper

    def update_bvh(self):
        """contact.py:672-677: edge boxes + refit, float32 mesh copy + refit.
        With ``bvh_rebuild_interval`` = k > 0 the hierarchies are rebuilt
        (new Morton order) every k-th call instead of refit."""
        self.compute_edge_aabbs()
        k = getattr(self, "bvh_rebuild_interval", 0)
        self._bvh_calls = getattr(self, "_bvh_calls", 0) + 1
        rebuild = k > 0 and self._bvh_calls % k == 0
        if rebuild:
            self.bvh_edges.rebuild()
        else:
            self.bvh_edges.refit()
        if self.has_triangles:
            self._triangle_aabbs()
            if rebuild:
                self.tri_mesh.rebuild()
            else:
                self.tri_mesh.refit()

    def _refit_edges(self):
        """The boxes the edge query reads, from x4 (after _pack)."""
        N.call("ipcb_lbvh_refit_edges", ctypes.byref(self.soup.c_struct()), N.ptr(self.x4),
               float(_thickness + buffer), ctypes.byref(self.bvh_edges._c), N.stream_handle())

    def _refit_triangles(self):
        """The boxes the point-triangle query reads, from x4 (after _pack)."""
        N.call("ipcb_lbvh_refit_triangles", ctypes.byref(self.soup.c_struct()), N.ptr(self.x4), 0.0,
               ctypes.byref(self.tri_mesh._c), N.stream_handle())

    def _refits_packed(self) -> bool:
        """Whether the packed boxes are all a detection has to form: not where
        update_bvh rebuilds or a subclass has its own boxes."""
        own = type(self).update_bvh is not ContactSolverBase.update_bvh or \
            type(self).compute_edge_aabbs is not ContactSolverBase.compute_edge_aabbs
        return not (own or getattr(self, "bvh_rebuild_interval", 0))

    def _refit_queries(self):
        """What the queries need of update_bvh: the packed boxes."""
        if not self._refits_packed():
            return self.update_bvh()
        self._pack()
        self._refit_edges()
        if self.has_triangles:
            self._refit_triangles()
        self._follow_x4()

    def _follow_x4(self):
        """After a detection (or a replay of one) that formed the packed boxes
        alone: box arrays and nodes follow from x4, as update_bvh forms them,
        when they are read."""
        if not self._refits_packed():
            return
        self.bvh_edges.follow(partial(_edge_aabbs, self.soup, self.x4, float(_thickness + buffer)))
        if self.has_triangles:
            self.tri_mesh.follow(partial(_triangle_aabbs, self.soup, self.x4))

    # ----------------------------------------------------------------- DCD
    def _grow_contact_list(self, contacts: Contacts, required: int, point_triangle: bool = False):
        """contact.py:523-537: grow to the next power of two."""
        contacts.grow(_next_pow2(required))
        if point_triangle:
            self.contacts_list_pt = contacts
        else:
            self.contacts_list_new = contacts
        if verbose:
            print(f"contact buffer grown to {contacts.capacity}")

    def _launch_dcd(self, which: str):
        soup = self.soup.c_struct()
        s = N.stream_handle()
        if which == "ee":
            self.contacts_new.cnt.zero_()
            N.call("ipcb_dcd_ee", ctypes.byref(soup), N.ptr(self.x4), ctypes.byref(self.bvh_edges._c),
                   float(_thickness), float(_thickness + buffer), int(self.disable_self_collision),
                   ctypes.byref(self.contacts_new.c_struct()), N.ptr(self._status), s)
        else:
            self.contacts_pt.cnt.zero_()
            N.call("ipcb_dcd_pt", ctypes.byref(soup), N.ptr(self.x4), ctypes.byref(self.tri_mesh._c),
                   float(_thickness), float(2.0 * (_thickness + buffer)), int(self.disable_self_collision),
                   N.ptr(self._point_order), ctypes.byref(self.contacts_pt.c_struct()), N.ptr(self._status), s)

    def _read_counts(self):
        """One host read of both list counts and the query status word (kept
        in ``query_status``)."""
        h = self._counts_host
        to = N.ptr(h)
        N.words((to, N.ptr(self.contacts_new.cnt)),
                (to + 4, N.ptr(self.contacts_pt.cnt) if self.has_triangles else None),
                (to + 8, N.ptr(self._status)))
        torch.cuda.current_stream().synchronize()
        self.query_status = int(h[2])
        return int(h[0]), int(h[1])

    def detect_collision(self):
        """contact.py:687-725.  Both queries are launched before the single
        count read; an overflowed list is grown and its query relaunched."""
        self.compute_V(ret=False)
        self._status.zero_()
        with self.profile_timer("collision BVH refit"):
            self._refit_queries()
        with self.profile_timer("EE collision query"):
            self._launch_dcd("ee")
        if self.has_triangles:
            with self.profile_timer("PT collision query"):
                self._launch_dcd("pt")
        with self.profile_timer("contact count host transfer"):
            n_ee, n_pt = self._read_counts()
        relaunched = False
        if n_ee > self.contacts_new.capacity:
            self._grow_contact_list(self.contacts_new, n_ee)
            self._launch_dcd("ee")
            relaunched = True
        if n_pt > self.contacts_pt.capacity:
            self._grow_contact_list(self.contacts_pt, n_pt, point_triangle=True)
            self._launch_dcd("pt")
            relaunched = True
        if relaunched:
            n_ee, n_pt = self._read_counts()
        self.n_contacts, self.n_contacts_pt = n_ee, (n_pt if self.has_triangles else 0)
        if self.query_status & QUERY_FAILED:
            warnings.warn(f"contact query ran out of its traversal bound (status {self.query_status}): "
                          "the candidate lists may be incomplete", RuntimeWarning, stacklevel=2)
        if verbose:
            print(f"n ee contacts = {self.n_contacts}\nn pt contacts = {self.n_contacts_pt}")

    # ----------------------------------------------------------------- CCD
    def collision_free_step(self, dx: torch.Tensor) -> float:
        """contact.py:539-585: conservative CCD bound for x -= alpha * dx;
        returns 0.9 * toi if toi < 1 else 1.  Leaves the swept boxes of the
        whole step in ccd_edge_lower / _upper and ccd_triangle_lower / _upper."""
        self._launch_ccd(dx)
        soup, s, x1 = ctypes.byref(self.soup.c_struct()), N.stream_handle(), N.ptr(self.ccd_x1)
        boxes = self.ccd_edge_lower, self.ccd_edge_upper
        N.call("ipcb_swept_edge_aabbs", soup, x1, 1e-7, *map(N.ptr, boxes), s)
        self.ccd_edge_bvh.follow(nodes=boxes)
        if self.has_triangles:
            boxes = self.ccd_triangle_lower, self.ccd_triangle_upper
            N.call("ipcb_swept_triangle_aabbs", soup, x1, 1e-7, *map(N.ptr, boxes), s)
            self.ccd_triangle_bvh.follow(nodes=boxes)
        return self._step_bound()

    def _step_bound(self) -> float:
        """One host read of the TOI and the query status.  The bound is
        0.9 * toi (1 when nothing collides), or 0 -- no step -- when a query
        set IPCB_STATUS_STACK or IPCB_STATUS_ROOT_ITERS: such a query may have
        missed an earlier impact, so its TOI is no bound.  Refusals are
        counted in ``ccd_refusals``."""
        h = self._counts_host
        toi, to, src = h[4:6] if self.ccd_toi.dtype == torch.float64 else h[4:5], N.ptr(h), N.ptr(self.ccd_toi)
        moves = [(to + 16 + 4 * k, src + 4 * k) for k in range(toi.numel())]
        N.words((to + 12, N.ptr(self._status)), *moves)
        torch.cuda.current_stream().synchronize()
        return self._bound_from(float(toi.view(self.ccd_toi.dtype)), int(h[3]))

    def _bound_from(self, toi: float, status: int) -> float:
        self.query_status = status
        if status & QUERY_FAILED:
            self.ccd_refusals += 1
            return 0.0
        return 0.9 * toi if toi < 1.0 else 1.0

    def _launch_ccd(self, dx: torch.Tensor, reset_status: bool = True):
        """The CCD queries of collision_free_step; the TOI stays in ccd_toi
        and the queries' status bits in _status (zeroed first unless
        reset_status is False)."""
        soup = self.soup.c_struct()
        s = N.stream_handle()
        N.call("ipcb_add_dx", ctypes.byref(soup), N.ptr(dx), N.ptr(self.ccd_x1), s)
        self.ccd_toi.fill_(1.0)
        if reset_status:
            self._status.zero_()
        if self.has_triangles:  # the two queries side by side, each with its own staging list
            if getattr(self, "_toi_ws_pt", None) is None:
                self._toi_ws_pt = torch.empty_like(self._toi_ws)
            with self._branch(0):
                self._ccd_query("pt", 0, self.soup.n_verts, self._toi_ws_pt)
        self._ccd_query("ee", 0, self.soup.n_edges, self._toi_ws)
        if self.has_triangles:
            self._join(0)

    def _ccd_query(self, which: str, first: int, count: int, ws: torch.Tensor):
        """One CCD query of the step x -> ccd_x1 on the current stream: boxes
        and TOI.  The contact list of the kind is tried first (whatever
        positions it was found at, its pairs are pairs of the query): the
        TOI it gives bounds the sweep the query has to look at."""
        soup = self.soup.c_struct()
        pad = 1e-7
        excl = int(self.disable_self_collision)
        s = N.stream_handle()
        if which == "ee":
            N.call("ipcb_edge_edge_step", ctypes.byref(soup), N.ptr(self.ccd_x1), pad,
                   ctypes.byref(self.ccd_edge_bvh._c), ctypes.byref(self.contacts_new.c_struct()), excl, first, count,
                   N.ptr(self.ccd_toi), N.ptr(self._status), N.ptr(ws), ws.numel(), s)
        else:
            N.call("ipcb_point_triangle_step", ctypes.byref(soup), N.ptr(self.ccd_x1), pad,
                   ctypes.byref(self.ccd_triangle_bvh._c), N.ptr(self._point_order),
                   ctypes.byref(self.contacts_pt.c_struct()), excl, first, count, N.ptr(self.ccd_toi),
                   N.ptr(self._status), N.ptr(ws), ws.numel(), s)

    def _both_queries(self, which: str, ws: torch.Tensor):
        """The discrete and the CCD query of one kind in one walk of its
        hierarchy (direction in ccd_x1): records into the contact list, the
        pairs that can touch within the step into ``ws``.  The caller has
        zeroed the list's count."""
        soup = self.soup.c_struct()
        pad = 1e-7
        excl = int(self.disable_self_collision)
        s = N.stream_handle()
        if which == "ee":
            N.call("ipcb_edge_edge_both", ctypes.byref(soup), N.ptr(self.ccd_x1), pad, ctypes.byref(self.bvh_edges._c),
                   float(_thickness), float(_thickness + buffer), excl, ctypes.byref(self.contacts_new.c_struct()),
                   N.ptr(self.ccd_toi), N.ptr(self._status), N.ptr(ws), ws.numel(), s)
        else:
            N.call("ipcb_point_triangle_both", ctypes.byref(soup), N.ptr(self.ccd_x1), pad,
                   ctypes.byref(self.tri_mesh._c), float(_thickness), float(2.0 * (_thickness + buffer)),
                   N.ptr(self._point_order), excl, ctypes.byref(self.contacts_pt.c_struct()), N.ptr(self.ccd_toi),
                   N.ptr(self._status), N.ptr(ws), ws.numel(), s)

    def _solve_staged(self, which: str, ws: torch.Tensor):
        """The TOI of the pairs _both_queries staged."""
        soup = self.soup.c_struct()
        pad = 1e-7
        excl = int(self.disable_self_collision)
        tail = (excl, N.ptr(self.ccd_toi), N.ptr(self._status), N.ptr(ws), ws.numel(), N.stream_handle())
        if which == "ee":
            N.call("ipcb_edge_edge_solve", ctypes.byref(soup), N.ptr(self.ccd_x1), pad,
                   ctypes.byref(self.ccd_edge_bvh._c), *tail)
        else:
            N.call("ipcb_point_triangle_solve", ctypes.byref(soup), N.ptr(self.ccd_x1), pad,
                   ctypes.byref(self.ccd_triangle_bvh._c), N.ptr(self._point_order), *tail)

    def new_intersections(self, x0: torch.Tensor, x1: torch.Tensor) -> float:
        """contact.py:587-670 (the augmented-Lagrangian solver's CCD): every
        EE / PT pair that collides on the straight path x0 -> x1 becomes a
        record of ``contacts_new`` / ``contacts_pt`` (alpha = its time of
        impact); returns 0.9 * toi if toi < 1 else 1.  Lists grow and the
        query reruns when they overflow, as the reference."""
        soup = self.soup.c_struct(x0)
        s = N.stream_handle()
        pad = 1e-7
        th = float(_thickness)
        excl = int(self.disable_self_collision)
        N.call("ipcb_swept_edge_aabbs", ctypes.byref(soup), N.ptr(x1), pad, N.ptr(self.ccd_edge_lower),
               N.ptr(self.ccd_edge_upper), s)
        self.ccd_edge_bvh.refit(self.ccd_edge_lower, self.ccd_edge_upper)
        self._status.zero_()

        def edges():
            self.contacts_new.cnt.zero_()
            self.ccd_toi.fill_(1.0)
            N.call("ipcb_edge_edge_intersections", ctypes.byref(soup), N.ptr(x1), ctypes.byref(self.ccd_edge_bvh._c),
                   N.ptr(self.ccd_edge_lower), N.ptr(self.ccd_edge_upper), excl, th, N.ptr(self.ccd_toi),
                   ctypes.byref(self.contacts_new.c_struct()), N.ptr(self._status), N.ptr(self._toi_ws),
                   self._toi_ws.numel(), s)
            return int(self.contacts_new.cnt.item())

        n = edges()
        if n > self.contacts_new.capacity:
            self._grow_contact_list(self.contacts_new, n)
            n = edges()
        self.n_contacts = n
        if self.has_triangles:
            N.call("ipcb_swept_triangle_aabbs", ctypes.byref(soup), N.ptr(x1), pad, N.ptr(self.ccd_triangle_lower),
                   N.ptr(self.ccd_triangle_upper), s)
            self.ccd_triangle_bvh.refit(self.ccd_triangle_lower, self.ccd_triangle_upper)

            def points():
                self.contacts_pt.cnt.zero_()
                N.call("ipcb_point_triangle_intersections", ctypes.byref(soup), N.ptr(x1),
                       ctypes.byref(self.ccd_triangle_bvh._c), pad, excl, th, N.ptr(self.ccd_toi),
                       ctypes.byref(self.contacts_pt.c_struct()), N.ptr(self._status), N.ptr(self._toi_ws),
                       self._toi_ws.numel(), s)
                return int(self.contacts_pt.cnt.item())

            n = points()
            if n > self.contacts_pt.capacity:
                self._grow_contact_list(self.contacts_pt, n, point_triangle=True)
                n = points()
            self.n_contacts_pt = n
        else:
            self.n_contacts_pt = 0
        return self._step_bound()

    def edge_triangle_crossings(self, capacity: int = 0):
        """Intersection check of the current positions: the number of
        (surface edge, surface triangle) pairs, without a shared vertex, whose
        segment crosses the triangle (an accepted IPC step leaves none), and
        up to ``capacity`` of them as an (m, 2) int32 tensor (edge,
        triangle).  Refits the triangle hierarchy to the positions (the next
        detect_collision refits it again)."""
        if not self.has_triangles:
            return 0, torch.zeros((0, 2), dtype=torch.int32, device=self.device)
        self._pack()
        self._triangle_aabbs()
        self.tri_mesh.refit()
        count = torch.zeros(1, dtype=torch.int32, device=self.device)
        pairs = torch.zeros((max(capacity, 1), 2), dtype=torch.int32, device=self.device)
        st = torch.zeros(1, dtype=torch.int32, device=self.device)
        N.call("ipcb_edge_triangle_crossings", ctypes.byref(self.soup.c_struct()), ctypes.byref(self.tri_mesh.c),
               N.ptr(count), N.ptr(pairs), int(capacity), N.ptr(st), N.stream_handle())
        n, status = (int(v) for v in torch.cat([count, st]).tolist())
        if status & QUERY_FAILED:
            raise RuntimeError(f"intersection check ran out of its traversal bound (status {status})")
        return n, pairs[:min(n, capacity)]

    @property
    def status(self) -> int:
        """OR of IPCB_STATUS_* bits raised by the last queries."""
        return int(self._status.item())
