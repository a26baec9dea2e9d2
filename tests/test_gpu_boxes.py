"""The public boxes, hierarchies and float positions after each call that
detects, although its queries form the packed boxes alone (gpu)."""
import numpy as np
import pytest
import torch

from ipc_warp_b200 import contact
from ipc_warp_b200.lbvh import Bvh
from ipc_warp_b200.newton import FEMContactSolver
from ipc_warp_b200.pipeline import ContactPipeline
from ipc_warp_b200.scenes import two_cubes

pytestmark = pytest.mark.gpu


def _scene():
    return two_cubes(n=4, gap=4e-4, angle_deg=15.0, jitter=0.0, seed=0, dhat=1e-3, kappa=1e6)


def _boxes(x, prims, pad):
    p = x[prims.cpu().numpy().reshape(len(prims), -1)]
    pad = np.float32(pad)
    return p.min(1) - pad, p.max(1) + pad


def _check(s, x):
    """Arrays, nodes and x4 of positions x (discrete boxes)."""
    x = x.float().cpu().numpy()
    assert np.array_equal(s.x4[:, :3].cpu().numpy(), x)
    for bvh, prims, pad, lo, hi in (
            (s.bvh_edges, s.soup.edges.view(-1, 2), contact._thickness + contact.buffer, s.bvh_edges_lower, s.bvh_edges_upper),
            (s.tri_mesh, s.soup.triangles.view(-1, 3), 0.0, s.tri_lower, s.tri_upper)):
        wl, wh = _boxes(x, prims, pad)
        assert np.array_equal(lo.cpu().numpy(), wl) and np.array_equal(hi.cpu().numpy(), wh)
        assert bvh.lower is lo and bvh.upper is hi
        root = bvh.nodes[0].cpu().numpy()
        assert np.array_equal(np.minimum(root[0, :3], root[2, :3]), wl.min(0))
        assert np.array_equal(np.maximum(root[1, :3], root[3, :3]), wh.max(0))


@pytest.mark.parametrize("call", ["detect_collision", "iteration", "iteration_host"])
def test_boxes_follow_a_detection(cuda, call):
    pipe = ContactPipeline.from_scene(_scene(), dtype=torch.float64, device=cuda)
    x0 = pipe.soup.x_transformed.clone()
    dx = torch.zeros_like(x0)
    for k in range(3):  # eager, captured, replayed
        x = x0 + 1e-5 * (k + 1)
        if call == "iteration_host":
            pipe.iteration_host(x.cpu().pin_memory(), dx.cpu().pin_memory(), torch.empty_like(x, device="cpu").pin_memory())
        else:
            pipe.soup.x_transformed.copy_(x)
            pipe.iteration(dx) if call == "iteration" else pipe.detect_collision()
        pipe.soup.x_transformed.add_(1.0)  # what is read later is of the detection
        _check(pipe, x)


def test_boxes_follow_solver_graphs(cuda):
    s = FEMContactSolver(_scene(), material="stvk", E=1e6, nu=0.4, rho=1000.0, h=1e-2, dtype=torch.float64)
    for k in range(3):
        s.states.x.add_(1e-5)
        s.compute_A()
        _check(s, s.states.x)
        s.states.dx.fill_(1e-6)
        assert s.line_search() > 0
        _check(s, s.states.x)


def test_swept_boxes_of_a_step(cuda):
    pipe = ContactPipeline.from_scene(_scene(), dtype=torch.float32, device=cuda)
    x = pipe.soup.x_transformed.cpu().numpy()
    pipe.detect_collision()
    dx = torch.full_like(pipe.soup.x_transformed, 0.25)
    pipe.collision_free_step(dx)
    for prims, lo, hi, bvh in (
            (pipe.soup.edges.view(-1, 2), pipe.ccd_edge_lower, pipe.ccd_edge_upper, pipe.ccd_edge_bvh),
            (pipe.soup.triangles.view(-1, 3), pipe.ccd_triangle_lower, pipe.ccd_triangle_upper, pipe.ccd_triangle_bvh)):
        (l0, h0), (l1, h1) = _boxes(x, prims, 0.0), _boxes(x - np.float32(0.25), prims, 0.0)
        assert np.allclose(lo.cpu().numpy(), np.minimum(l0, l1), atol=1e-6)
        assert np.allclose(hi.cpu().numpy(), np.maximum(h0, h1), atol=1e-6)
        root = bvh.nodes[0].cpu().numpy()
        assert np.array_equal(np.minimum(root[0, :3], root[2, :3]), lo.cpu().numpy().min(0))
    wl, _ = _boxes(x, pipe.soup.edges.view(-1, 2), contact._thickness + contact.buffer)
    assert np.array_equal(pipe.bvh_edges_lower.cpu().numpy(), wl)  # still the detection's


class Wider(FEMContactSolver):
    """A subclass with its own boxes."""
    calls = 0

    def update_bvh(self):
        self.calls += 1
        super().update_bvh()


def test_overridden_update_is_called(cuda):
    s = Wider(_scene(), material="stvk", E=1e6, nu=0.4, rho=1000.0, h=1e-2, dtype=torch.float64)
    ref = FEMContactSolver(_scene(), material="stvk", E=1e6, nu=0.4, rho=1000.0, h=1e-2, dtype=torch.float64)
    for call in ("detect_collision", "compute_A", "line_search", "compute_collision_energy"):
        before = s.calls
        getattr(s, call)()
        getattr(ref, call)()
        assert s.calls > before, call
    assert (s.n_contacts, s.n_contacts_pt) == (ref.n_contacts, ref.n_contacts_pt) and s.n_contacts > 0


def test_hierarchy_forms_boxes_once_read(cuda):
    lo = torch.rand(100, 3, device=cuda)
    bvh = Bvh(lo, lo + 0.1)
    formed = []
    bvh.follow(lambda a, b: (formed.append(1), a.copy_(lo + 1), b.copy_(lo + 1)))
    other = (lo + 5, lo + 6)
    bvh.follow(nodes=other)
    assert float(bvh.nodes[0, 0, 0]) >= 5 and not formed  # the nodes' own boxes
    assert bvh.lower is not None and formed == [1]
    bvh.refit()
    assert formed == [1]
