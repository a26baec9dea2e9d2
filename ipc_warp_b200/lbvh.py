"""Linear BVH over AABB arrays: the stand-in for ``wp.Bvh`` / ``wp.Mesh``
(contact.py:464-483: built once, ``.refit()`` per query, contact.py:672-677).

``Bvh(lower, upper)`` keeps references to the two float32 (n, 3) box tensors
like ``wp.Bvh`` does, builds the hierarchy on construction (Morton codes,
device radix sort, Karras emission, atomic refit) and exposes ``refit()``
(same topology, new boxes) and ``rebuild()`` (new topology).
"""
from __future__ import annotations

import ctypes

import torch

from . import _native as N


class Bvh:
    def __init__(self, lower: torch.Tensor, upper: torch.Tensor, capacity: int | None = None):
        assert lower.dtype == torch.float32 and upper.dtype == torch.float32
        assert lower.shape == upper.shape and lower.shape[-1] == 3
        self._lower, self._upper = lower, upper
        self._form = self._nodes_of = None
        self.device = lower.device
        n = lower.shape[0]
        self.capacity = max(int(capacity or n), 1)
        self._mem = torch.empty(N.size("ipcb_lbvh_bytes", self.capacity), dtype=torch.uint8, device=self.device)
        self._ws = torch.empty(N.size("ipcb_lbvh_build_workspace", self.capacity), dtype=torch.uint8,
                               device=self.device)
        self._c = N.Lbvh()
        N.call("ipcb_lbvh_bind", ctypes.byref(self._c), N.ptr(self._mem), self.capacity)
        self.rebuild()

    def follow(self, form=None, nodes=None) -> None:
        """The packed boxes (what the queries walk) have been formed from
        positions alone.  form(lower, upper) brings the bound box arrays up to
        them once somebody reads those, and the nodes are refit to ``nodes``, a
        (lower, upper) pair (default: the bound arrays), once somebody reads
        them."""
        if form is not None:
            self._form = form
        self._nodes_of = (self._lower, self._upper) if nodes is None else nodes

    def settle_boxes(self) -> None:
        if self._form is not None:
            form, self._form = self._form, None
            form(self._lower, self._upper)

    def rewrite(self) -> tuple[torch.Tensor, torch.Tensor]:
        """The bound box arrays, for a caller that writes all of them."""
        self._form = None
        return self._lower, self._upper

    @property
    def c(self) -> N.Lbvh:
        """The C structure, its nodes up to date (``_c``: for the queries of
        the packed boxes)."""
        if self._nodes_of is not None:
            if self._nodes_of[0] is self._lower:
                self.settle_boxes()
            self.refit(*self._nodes_of)
        return self._c

    @property
    def lower(self) -> torch.Tensor:
        self.settle_boxes()
        return self._lower

    @lower.setter
    def lower(self, boxes: torch.Tensor):
        self.settle_boxes()
        self._lower = boxes

    @property
    def upper(self) -> torch.Tensor:
        self.settle_boxes()
        return self._upper

    @upper.setter
    def upper(self, boxes: torch.Tensor):
        self.settle_boxes()
        self._upper = boxes

    @property
    def n(self) -> int:
        return self._c.n

    def _view(self, addr: int, count: int, dtype=torch.int32) -> torch.Tensor:
        off = addr - self._mem.data_ptr()
        nbytes = count * torch.tensor([], dtype=dtype).element_size()
        return self._mem[off:off + nbytes].view(dtype)

    @property
    def sorted(self) -> torch.Tensor:
        """Primitive of each leaf slot (Morton order), int32[n]."""
        return self._view(self._c.sorted, self._c.n)

    @property
    def nodes(self) -> torch.Tensor:
        """Internal nodes as float32[n-1, 4, 4]: (L.lo, Lcode) (L.hi) (R.lo, Rcode) (R.hi)."""
        m = max(self.c.n - 1, 1)
        return self._view(self.c.nodes, 16 * m, torch.float32).view(m, 4, 4)

    @property
    def parent(self) -> torch.Tensor:
        return self._view(self._c.parent, 2 * self.capacity)

    def rebuild(self, lower: torch.Tensor | None = None, upper: torch.Tensor | None = None, stream=None):
        if lower is not None:
            self._lower, self._upper, self._form = lower, upper, None
        self.settle_boxes()
        self._nodes_of = None
        n = self._lower.shape[0]
        if n > self.capacity:
            raise ValueError(f"Bvh capacity {self.capacity} < {n} boxes")
        N.call("ipcb_lbvh_build", ctypes.byref(self._c), N.ptr(self._lower), N.ptr(self._upper), n,
               N.ptr(self._ws), self._ws.numel(), N.stream_handle(stream))

    def refit(self, lower: torch.Tensor | None = None, upper: torch.Tensor | None = None, stream=None):
        """Recompute node boxes keeping the topology; by default from the
        bound box arrays, or from other (n, 3) boxes of the same primitives."""
        lo = self.lower if lower is None else lower
        hi = self.upper if upper is None else upper
        self._nodes_of = None
        assert lo.shape[0] == self._c.n and hi.shape[0] == self._c.n
        N.call("ipcb_lbvh_refit", ctypes.byref(self._c), N.ptr(lo), N.ptr(hi), N.stream_handle(stream))


def sort_pairs(keys: torch.Tensor, vals: torch.Tensor, end_bit: int, stream=None) -> None:
    """In-place stable device radix sort of (keys, vals) by the low end_bit bits."""
    n = keys.numel()
    if keys.dtype == torch.int32:
        ws = torch.empty(N.size("ipcb_sort_workspace_u32", n), dtype=torch.uint8, device=keys.device)
        N.call("ipcb_sort_pairs_u32", N.ptr(keys), N.ptr(vals), n, end_bit, N.ptr(ws), ws.numel(),
               N.stream_handle(stream))
    elif keys.dtype == torch.int64:
        ws = torch.empty(N.size("ipcb_sort_workspace_u64", n), dtype=torch.uint8, device=keys.device)
        N.call("ipcb_sort_pairs_u64", N.ptr(keys), N.ptr(vals), n, end_bit, N.ptr(ws), ws.numel(),
               N.stream_handle(stream))
    else:
        raise TypeError(keys.dtype)
