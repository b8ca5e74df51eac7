"""The sort's look-back over batches of tiles, at tile counts around its batches: a stable sort has one
result, so it must equal NumPy's."""
import ctypes as C

import numpy as np
import pytest

from splishsplash_for_cuda_b200 import _capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", [1, 2, 4, 5, 6, 8, 9, 10, 37])
@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_tile_counts(tiles, extra):
    import torch

    n = 2048 * tiles + extra
    rng = np.random.default_rng(n)
    keys = (rng.integers(0, 1 << 12, n) * rng.integers(1, 1 << 10, n)).astype(np.uint32)  # many duplicates
    dev = torch.device("cuda", 0)
    k = torch.from_numpy(keys.view(np.int32)).to(dev)
    ko, po = torch.empty_like(k), torch.empty_like(k)
    code = _capi.load().dfsph_sort_cell_keys_noalloc(C.c_void_p(k.data_ptr()), C.c_void_p(ko.data_ptr()),
                                                     C.c_void_p(po.data_ptr()), n, 24,
                                                     C.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
    assert code == _capi.DFSPH_OK
    ref = np.argsort(keys, kind="stable")
    assert np.array_equal(po.cpu().numpy(), ref) and np.array_equal(ko.cpu().numpy().view(np.uint32), keys[ref])
