"""Rows of every register count of the assembly's row sort, their runs and
the order of their sums (gpu)."""
import numpy as np
import pytest
import torch

from ipc_warp_b200.bsr import bsr_from_triplets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("columns", [1, 7, 2000])
def test_row_lengths_at_the_edges(cuda, columns, fp64):
    lengths = [0, 1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 3, 0]
    rng = np.random.default_rng(columns)
    dt = np.float64 if fp64 else np.float32
    rows = np.concatenate([np.full(L, r) for r, L in enumerate(lengths)]).astype(np.int32)
    cols = rng.integers(0, columns, size=len(rows)).astype(np.int32)
    cols[rows == 8] = 5 % columns  # one run over several registers
    vals = rng.normal(size=(len(rows), 3, 3)).astype(dt)
    mix = rng.permutation(len(rows))
    rows, cols, vals = rows[mix], cols[mix], vals[mix]
    A = bsr_from_triplets(len(lengths), 2000, *(torch.tensor(a, device=cuda) for a in (rows, cols, vals)))
    off, n = A.offsets.cpu().numpy(), A.nnz_sync()
    got_c, got_v = A.columns[:n].cpu().numpy(), A.values[:n].cpu().numpy()
    for r in range(len(lengths)):
        mine = rows == r
        want = np.unique(cols[mine])
        assert np.array_equal(got_c[off[r]:off[r + 1]], want)
        for u, c in enumerate(want):
            block = vals[mine & (cols == c)].astype(np.float64)
            # m summands in any order: (m - 1) roundings of partial sums
            tol = len(block) * np.finfo(dt).eps * np.abs(block).sum(axis=0)
            assert np.all(np.abs(got_v[off[r] + u] - block.sum(axis=0)) <= tol)
