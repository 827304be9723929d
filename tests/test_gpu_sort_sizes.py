"""The pair sort across its forms: one launch up to 65,536 pairs (a thread one
to eight pairs, one to sixteen CTAs), three kernels a pass beyond, odd and even
pass counts in place, digits that all keys share, many ties; against a stable
key sort."""
import ctypes

import numpy as np
import pytest

from fluidgrid_gb300 import _ffi, build

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SIZES = [1, 31, 1023, 1024, 1025, 8191, 8192, 8193, 16384, 16385, 32767, 32769, 65535, 65536, 65537, 70001, 300007]


@pytest.mark.parametrize("n", SIZES)
def test_sorts_are_stable(n):
    build.build()
    L = _ffi.load()
    rng = np.random.default_rng(n)
    for bits, keys in ((32, rng.integers(0, 1 << 32, n, dtype=np.uint64)),
                       (32, rng.integers(0, 700, n, dtype=np.uint64)),
                       (32, np.full(n, 0xffffffff, np.uint64)),
                       (32, 0xffffff00 + rng.integers(0, 256, n, dtype=np.uint64)),
                       (21, rng.integers(0, 1 << 32, n, dtype=np.uint64)),
                       (17, rng.integers(0, 1 << 17, n, dtype=np.uint64)),
                       (8, rng.integers(0, 5, n, dtype=np.uint64)),
                       (1, rng.integers(0, 1 << 32, n, dtype=np.uint64)),
                       (0, rng.integers(0, 1 << 32, n, dtype=np.uint64))):
        k = keys.astype(np.uint32)
        v = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
        order = np.argsort(k.astype(np.uint64) & ((1 << bits) - 1), kind="stable")
        for api in ("fgc_sort_pairs", "fg_sort_pairs_noalloc", "gSort"):
            if api == "gSort" and bits != 32:
                continue
            kt, vt = torch.from_numpy(k.view(np.int32)).cuda(), torch.from_numpy(v.view(np.int32)).cuda()
            a, b = ctypes.c_void_p(kt.data_ptr()), ctypes.c_void_p(vt.data_ptr())
            if api == "gSort":
                L.gSort(a, b, n)
            elif api == "fgc_sort_pairs":
                L.fgc_sort_pairs(a, b, bits, n)
            else:
                assert L.fg_sort_pairs_noalloc(a, b, bits, n, None) == 0
            assert api == "fg_sort_pairs_noalloc" or L.fgc_last_status() == 0
            assert np.array_equal(kt.cpu().numpy().view(np.uint32), k[order]), (api, bits)
            assert np.array_equal(vt.cpu().numpy().view(np.uint32), v[order]), (api, bits)
