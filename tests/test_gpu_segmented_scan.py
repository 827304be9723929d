"""fgc_segmented_scan_float4 over sizes: one chunk to more than a cluster's
round of chunks, flags nowhere, everywhere and at the chunks' edges, in place;
whole-number inputs, whose sums are exact in any order."""
import ctypes

import numpy as np
import pytest

from fluidgrid_gb300 import _ffi, build

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1024, 1025, 2049, 8191, 8192, 8193, 20001])
def test_segmented_scan(n):
    build.build()
    L = _ffi.load()
    rng = np.random.default_rng(n)
    x = rng.integers(-40, 41, (n, 4)).astype(np.float32)
    edges = np.zeros(n, np.uint32)
    edges[np.arange(0, n, 1024)] = 7
    edges[np.arange(1023, n, 1024)] = 1
    for flags in (np.zeros(n, np.uint32), np.ones(n, np.uint32), edges,
                  (rng.random(n) < 0.001).astype(np.uint32), (rng.random(n) < 0.2).astype(np.uint32)):
        total = np.cumsum(x.astype(np.int64), 0)
        head = np.maximum.accumulate(np.where(flags != 0, np.arange(n), -1))
        before = np.where(head[:, None] > 0, total[np.maximum(head - 1, 0)], 0)
        want = (total - before).astype(np.float32)
        f = torch.from_numpy(flags.view(np.int32)).cuda()
        for inplace in (False, True):
            a = torch.from_numpy(x).cuda()
            out = a if inplace else torch.empty_like(a)
            L.fgc_segmented_scan_float4(ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(a.data_ptr()),
                                        ctypes.c_void_p(f.data_ptr()), n)
            assert L.fgc_last_status() == 0
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy(), want)
