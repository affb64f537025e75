"""Exact SVD whose output overlaps its input: U over A for tall blocks, V^T over A for flat ones, in every form (one
CTA, clusters that hold the block, clusters that go through L2, the cooperative grid).  Results must equal the ones of
separate buffers bit by bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(40, 20), (120, 90), (3000, 400), (1300, 512), (20, 40), (90, 120), (400, 3000), (512, 1300)])
def test_an_output_may_overlap_the_input(m, n):
    from xped_gb300 import ensure_device, lib
    from xped_gb300._lib import SvdDesc, last_error
    ensure_device(0)
    L = lib()
    k = min(m, n)
    d = (SvdDesc * 1)(SvdDesc(m=m, n=n))
    a = np.random.default_rng(m).standard_normal((n, m)) * np.logspace(0, -3, m)  # column-major, graded rows
    size = {"a": 8 * m * n, "u": 8 * m * k, "s": 8 * k, "v": 8 * k * n, "w": L.xgb_svd_workspace_bytes(1, d)}
    ptr = {}
    for name, nbytes in size.items():
        ptr[name] = C.c_void_p()
        assert L.xgb_malloc(C.byref(ptr[name]), nbytes) == 0
    results = []
    for over in (None, "u" if m >= n else "v"):
        at = dict(ptr)
        if over:
            at[over] = ptr["a"]
        assert L.xgb_memcpy_h2d(ptr["a"], a.ctypes.data, a.nbytes) == 0
        assert L.xgb_batched_svd(1, d, at["a"], at["u"], at["s"], at["v"], at["w"], None) == 0, last_error()
        out = []
        for name in "usv":
            x = np.empty(size[name] // 8)
            assert L.xgb_memcpy_d2h(x.ctypes.data, at[name], x.nbytes) == 0
            out.append(x)
        results.append(out)
    for p in ptr.values():
        L.xgb_free(p)
    for x, y in zip(*results):
        assert np.array_equal(x, y)
