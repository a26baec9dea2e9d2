"""The PCG's iterations on the sliced copy of the matrix (ipcb_pcg_slice):
rows of every length around the slices' bounds, rows above them, row counts
around a window, and solves that end inside, at and after a batch (gpu)."""
import numpy as np
import pytest
import torch

from ipc_warp_b200.bsr import BsrMatrix
from ipc_warp_b200.newton import BlockJacobi, DevicePcg, JacobiPrecond, pcg

pytestmark = pytest.mark.gpu


def spd(n, long_rows, dtype, seed, device):
    """A symmetric positive definite block matrix: a random graph plus
    ``long_rows`` hubs joined to a large part of the vertices."""
    rng = np.random.default_rng(seed)
    pairs = {(int(a), int(b)) for a, b in rng.integers(0, n, size=(3 * n, 2)) if a < b}
    for h in range(long_rows):
        pairs |= {(min(h, int(j)), max(h, int(j))) for j in rng.integers(0, n, size=n // 2) if j != h}
    blocks = {(i, i): np.eye(3) * rng.uniform(0.05, 1.0) for i in range(n)}
    for a, b in sorted(pairs):
        g = rng.normal(size=(3, 3))
        g = g @ g.T
        blocks[a, b] = blocks[b, a] = -g
        blocks[a, a] = blocks[a, a] + g
        blocks[b, b] = blocks[b, b] + g
    keys = sorted(blocks)
    A = BsrMatrix(n, n, len(keys), dtype, device)
    rows = np.array([k[0] for k in keys])
    A.offsets.copy_(torch.from_numpy(np.searchsorted(rows, np.arange(n + 1)).astype(np.int32)))
    A.columns.copy_(torch.tensor([k[1] for k in keys], dtype=torch.int32))
    A.values.copy_(torch.from_numpy(np.stack([blocks[k] for k in keys])))
    A.nnz_dev.fill_(len(keys))
    return A


@pytest.mark.parametrize("n,hubs", [(1, 0), (31, 0), (256, 1), (257, 3), (700, 2)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_sliced_iterations_match_host_pcg(cuda, n, hubs, dtype):
    A = spd(n, hubs, dtype, n, cuda)
    if hubs:
        lens = A.offsets[1:] - A.offsets[:-1]
        assert int(lens.max()) > 64 and int(lens.min()) >= 1
    b = torch.randn((n, 3), device=cuda, dtype=dtype)
    # float32 residuals drift from the recursion's: the tolerance is kept well above its rounding
    tol = 1e-4 if dtype == torch.float32 else 1e-10
    xh, ih, _ = pcg(A, b, BlockJacobi(A), tol, 5000)
    for use_graph in (False, True):
        x, it, rel, status = DevicePcg(batch=2, use_graph=use_graph).solve(A, b, JacobiPrecond(A), tol, 5000)
        assert status == 0 and rel <= tol and abs(it - ih) <= max(2, ih // 20)
        # both stop at |r| <= tol |b|; A's smallest eigenvalue is at least 0.05
        assert float((x - xh).double().norm()) <= 2.5 * tol * float(b.double().norm()) / 0.05
    for most in (1, 2, 3, 5, 6, 7):  # inside and at the ends of the batches of 2 and 4
        if most >= ih:
            break
        x, it, rel, status = DevicePcg(batch=2).solve(A, b, JacobiPrecond(A), 0.0, most)
        xm, im, relm = pcg(A, b, BlockJacobi(A), 0.0, most)
        assert it == im == most and status == 0
        # the same iterates, rounded in another order
        assert float((x - xm).double().norm()) <= (1e-3 if dtype == torch.float32 else 1e-9) * float(xm.double().norm())


def test_indefinite_matrix_breaks_down_after_the_copy(cuda):
    A = spd(300, 0, torch.float64, 1, cuda)
    rows = torch.repeat_interleave(torch.arange(300, device=cuda), (A.offsets[1:] - A.offsets[:-1]).long())
    diag = (rows == A.columns).nonzero().view(-1)
    A.values[diag[7]] = -A.values[diag[7]]
    b = torch.randn((300, 3), device=cuda, dtype=torch.float64)
    eye = JacobiPrecond(A)
    eye.dinv.copy_(torch.eye(3, dtype=torch.float64, device=cuda).expand(300, 3, 3))
    few = DevicePcg(batch=1).solve(A, b, eye, 1e-12, 5000)
    many = DevicePcg(batch=512).solve(A, b, eye, 1e-12, 5000)  # block-row order throughout
    assert few[3] & 1 and many[3] & 1 and abs(few[1] - many[1]) <= 1
