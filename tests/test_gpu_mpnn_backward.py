"""Parameter gradients of the learned preconditioner's net against the same
backward pass in float64, at row counts around the 128-row tiles, a hub row,
several tiles a CTA, and a gradient buffer off the vector alignment (gpu)."""
import numpy as np
import pytest
import torch

from ipc_warp_b200 import learned as L
from oracle import mpnn as om
from test_gpu_mpnn import _bsr

pytestmark = pytest.mark.gpu


def _system(nb, hub, cuda):
    offsets, cols, vals = om.random_spd(nb, nb)
    if hub:  # vertex 0 joined to all others
        rows = np.repeat(np.arange(nb), np.diff(offsets))
        blocks = {(int(i), int(j)): v for i, j, v in zip(rows, cols, vals)}
        for j in range(1, nb):
            for k in ((0, j), (j, 0)):
                blocks[k] = blocks.get(k, 0.0) - 0.1 * np.eye(3)
            blocks[0, 0] = blocks[0, 0] + 0.2 * np.eye(3)
            blocks[j, j] = blocks[j, j] + 0.2 * np.eye(3)
        keys = sorted(blocks)
        offsets = np.searchsorted([k[0] for k in keys], np.arange(nb + 1))
        cols, vals = np.array([k[1] for k in keys]), np.stack([blocks[k] for k in keys])
    return L.System.from_bsr(_bsr(offsets, cols, vals, torch.float32, cuda))


def _reference(sysm, net, tape, dG):
    """The gradients in float64 on the tape's activations, and the sums of
    the magnitudes of their terms."""
    g, dev = sysm.graph, sysm.A.device
    p = {k: torch.tensor(np.asarray(v), device=dev) for k, v in L.unflatten(net.params.cpu().numpy()).items()}
    w = {k: v.bfloat16().double() for k, v in p.items()}
    rows, cols, lower = g.rows.long(), g.columns[:g.nnz].long(), g.lower.long()
    deg = (g.offsets[1:] - g.offsets[:-1]).double()
    h, e, m, a, u = (t.double() for t in (tape.h, tape.e, tape.m, tape.a, tape.u))
    rnd = lambda t: t.bfloat16().double()
    grads, mags = {}, {}

    def add(wk, bk, X, dY):
        grads[wk], grads[bk] = X.T @ dY, dY.sum(0)
        mags[wk], mags[bk] = X.abs().T @ dY.abs(), dY.abs().sum(0)

    dout = dG.double()[:, :9]
    add("W_off", "b_off", e[L.LAYERS][lower], dout)
    de = torch.zeros((g.nnz, L.WIDTH), dtype=torch.float64, device=dev)
    de[lower] = dout @ w["W_off"].T
    dh = torch.zeros((g.n, L.WIDTH), dtype=torch.float64, device=dev)
    for l in reversed(range(L.LAYERS)):
        du = rnd(dh * (u[l] > 0))
        add(f"W2_{l}", f"b2_{l}", torch.cat([h[l], a[l]], 1), du)
        dXn = du @ w[f"W2_{l}"].T
        dm = rnd((de + (dXn[:, L.WIDTH:] / deg[:, None])[rows]) * (m[l] > 0))
        add(f"W1_{l}", f"b1_{l}", torch.cat([h[l][rows], h[l][cols], e[l]], 1), dm)
        dX = dm @ w[f"W1_{l}"].T
        dh = dh + dXn[:, :L.WIDTH]
        dh.index_add_(0, rows, dX[:, :L.WIDTH])
        dh.index_add_(0, cols, dX[:, L.WIDTH:2 * L.WIDTH])
        de = de + dX[:, 2 * L.WIDTH:]
    add("W_hin", "b_hin", sysm.x.double(), rnd(dh * (h[0] > 0)))
    add("W_ein", "b_ein", sysm.y.double(), rnd(de * (e[0] > 0)))
    return grads, mags


@pytest.mark.parametrize("nb,hub,shift", [(1, False, 0), (2, False, 1), (31, False, 0), (128, False, 0),
                                          (129, True, 0), (2500, True, 3), (20000, False, 0)])
def test_gradients_match_float64(cuda, nb, hub, shift):
    sysm = _system(nb, hub, cuda)
    net = L.Net(L.flatten(om.init_params(7, zero_head=False)), device=cuda)
    H, tape = L.forward(net, sysm, training=True)
    dG = torch.zeros((sysm.graph.n_lower, 64), dtype=torch.bfloat16, device=cuda)
    dG[:, :9] = torch.randn((sysm.graph.n_lower, 9), generator=torch.Generator(cuda).manual_seed(nb), device=cuda)
    grad = torch.ones(net.params.numel() + shift, device=cuda)[shift:]  # the gradients are added
    L.backward(net, sysm, tape, dG, grad)
    got = L.unflatten((grad.double() - 1.0).cpu().numpy())
    ref, mag = _reference(sysm, net, tape, dG)
    for k, _ in L.PARAMS:
        r, s = ref[k].cpu().numpy().ravel(), mag[k].cpu().numpy().ravel()
        # sums rounded in another order can flip the bf16 rounding of a gradient (2^-8 of
        # it), which is then a small part of a sum; the buffer's ones cost 2^-24 each add
        err = np.linalg.norm(np.asarray(got[k]).ravel() - r)
        assert err <= 2.0 ** -8 * np.linalg.norm(s) + 1e-4, (k, err, np.linalg.norm(s))
        if nb > 100 and np.linalg.norm(r) > 0:
            assert err <= 2.0 ** -6 * np.linalg.norm(r) + 1e-4, (k, err, np.linalg.norm(r))
