"""Row packing (pb_rows_compact) against numpy indexing: bytes are equal."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cap", [(1, 1), (1, 40), (7, 33), (9, 31), (300, 5), (40000, 3)])
def test_rows_are_packed_in_history_order(n, cap, cuda_device):
    import torch

    from pyrite_b200 import _lib as L
    from pyrite_b200.api import _Holder, _row_block

    rng = np.random.default_rng(n * 100 + cap)
    counts = rng.integers(0, cap + 1, n)
    counts[0] = cap
    h = _Holder(cuda_device)
    src, block, parts = _row_block(h, n * cap)
    block.copy_(torch.from_numpy(rng.integers(0, 256, block.numel(), dtype=np.uint8)))
    dst, packed, out = _row_block(h, int(counts.sum()))
    c = torch.from_numpy(counts).to(cuda_device)
    off = torch.from_numpy(np.cumsum(counts) - counts).to(cuda_device)
    L.check(L.load().pb_rows_compact(C.byref(src), n, cap, c.data_ptr(), off.data_ptr(), C.byref(dst), None),
            "pb_rows_compact")
    torch.cuda.synchronize(cuda_device)
    keep = (np.arange(cap)[None, :] < counts[:, None]).reshape(-1)
    a, b = block.cpu().numpy(), packed.cpu().numpy()
    for (key, o, nb, _t, _s), (_k, o2, nb2, _t2, _s2) in zip(parts, out):
        ref = a[o:o + nb].reshape(n * cap, -1)[keep]
        assert np.array_equal(b[o2:o2 + nb2], ref.reshape(-1)), key
