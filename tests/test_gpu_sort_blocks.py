"""The entry sort around the sizes where its blocks change (B200 required):
a quarter block, and the last size sorted in quarter blocks, against numpy's
stable sort.  Whole numbers: exactly equal."""
import ctypes as C

import numpy as np
import pytest

from splat_b200 import native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [8, 16])
@pytest.mark.parametrize("n", [1023, 1024, 1025, 4097, 262143, 262144, 262145])
def test_sort_at_block_sizes(n, bits):
    import torch
    rng = np.random.default_rng(n + bits)
    k = rng.integers(0, 1 << bits, n).astype(np.uint32)
    k[: n // 3] = 7  # long runs of one digit
    v = np.arange(n, dtype=np.uint32)
    dk, dv = torch.from_numpy(k.view(np.int32)).cuda(), torch.from_numpy(v.view(np.int32)).cuda()
    torch.cuda.synchronize()
    N.check(N.lib().gs_sort_entries_static(C.c_void_p(dk.data_ptr()), C.c_void_p(dv.data_ptr()), n, bits, None))
    order = np.argsort(k, kind="stable")
    assert np.array_equal(dk.cpu().numpy().view(np.uint32), k[order])
    assert np.array_equal(dv.cpu().numpy().view(np.uint32), v[order])
