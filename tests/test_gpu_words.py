"""Counters reset and read through ipcb_words (gpu)."""
import pytest
import torch

from ipc_warp_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 7, 8])
def test_words_move_and_reset(cuda, n):
    src = torch.arange(100, 116, dtype=torch.int32, device=cuda)
    dst = torch.full((16,), -1, dtype=torch.int32).pin_memory()
    moves = [(N.ptr(dst) + 8 * k, None if k % 3 == 2 else N.ptr(src) + 4 * k) for k in range(n)]
    N.words(*moves)
    torch.cuda.synchronize()
    want = [-1] * 16
    for k in range(n):
        want[2 * k] = 0 if k % 3 == 2 else 100 + k
    assert dst.tolist() == want


def test_words_refuses_more_and_null(cuda):
    w = torch.zeros(16, dtype=torch.int32, device=cuda)
    with pytest.raises(N.NativeError):
        N.words(*[(N.ptr(w) + 4 * k, None) for k in range(9)])
    with pytest.raises(N.NativeError):
        N.words((None, N.ptr(w)))
