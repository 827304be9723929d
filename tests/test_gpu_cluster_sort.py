"""The one-launch sort with every size of cluster that a GPU, or a part of one,
may place (one to sixteen CTAs, one to eight pairs a thread), against a stable
sort."""
import ctypes

import numpy as np
import pytest

from fluidgrid_gb300 import _ffi, build

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def L():
    build.build()
    return _ffi.load()


def pairs(n, bits, seed):
    rng = np.random.default_rng(seed)
    k = rng.integers(0, 1 << min(bits, 32), n, dtype=np.uint64).astype(np.uint32)
    k[: n // 3] = k[n // 2] if n > 2 else k[0]
    return k, rng.permutation(n).astype(np.uint32)


@pytest.mark.parametrize("ctas", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("bits", [5, 17, 32])
def test_every_cluster_size(L, ctas, bits):
    for n in (1, 1023, 1024 * ctas, 1024 * ctas + 1, 4096 * ctas, 4096 * ctas + 1, 8192 * ctas - 7, 8192 * ctas):
        if n > 65536:
            continue
        k, v = pairs(n, bits, n)
        order = np.argsort(k.astype(np.uint64) & ((1 << bits) - 1), kind="stable")
        kt, vt = torch.from_numpy(k.view(np.int32)).cuda(), torch.from_numpy(v.view(np.int32)).cuda()
        assert L.fg_selftest_cluster_sort(ctas, ctypes.c_void_p(kt.data_ptr()), ctypes.c_void_p(vt.data_ptr()), bits,
                                          n, None) == 0, L.fg_last_error()
        assert np.array_equal(kt.cpu().numpy().view(np.uint32), k[order]), n
        assert np.array_equal(vt.cpu().numpy().view(np.uint32), v[order]), n


def test_refused(L):
    t = torch.zeros(16, dtype=torch.int32, device="cuda")
    p = ctypes.c_void_p(t.data_ptr())
    for ctas, bits, n in ((0, 8, 8), (3, 8, 8), (32, 8, 8), (1, 0, 8), (1, 33, 8), (1, 8, 0), (1, 8, 8193),
                          (16, 8, 65537)):
        assert L.fg_selftest_cluster_sort(ctas, p, p, bits, n, None) == 1, (ctas, bits, n)

