"""FP64-accurate tensor-core products of few rows and columns over a long k (a full contraction is 1 x 1): against numpy to
the bound of the slicing, 2^-49 k max|a_i| max|b_j| with a factor of 8, and the time of one, which its slicing must not
keep on eight SMs."""
import ctypes as C
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F64TC = 4


def product(m, n, k, ta, tb, rng):
    from xped_gb300 import ensure_device, lib
    from xped_gb300._lib import GemmDesc, last_error
    ensure_device(0)
    L = lib()
    a, b = rng.standard_normal((m, k)) * np.exp(rng.uniform(-9, 0, (m, 1))), rng.standard_normal((k, n))
    a[:, k // 2:] *= 1e-3  # the largest entry of a row lies in its first half
    d = (GemmDesc * 1)(GemmDesc(m=m, n=n, k=k, lda=k if ta else m, ldb=n if tb else k, ldc=m, trans_a=ta, trans_b=tb))
    ptr = []
    for x in (a if ta else a.T, b if tb else b.T, np.zeros((n, m))):
        x = np.ascontiguousarray(x)
        p = C.c_void_p()
        assert L.xgb_malloc(C.byref(p), x.nbytes) == 0
        assert L.xgb_memcpy_h2d(p, x.ctypes.data, x.nbytes) == 0
        ptr.append(p)
    best = 1e9
    for _ in range(6):
        L.xgb_synchronize()
        t0 = time.perf_counter()
        assert L.xgb_grouped_gemm(F64TC, 1, d, *ptr, 1.0, 0.0, None) == 0, last_error()
        L.xgb_synchronize()
        best = min(best, time.perf_counter() - t0)
    c = np.empty((n, m))
    assert L.xgb_memcpy_d2h(c.ctypes.data, ptr[2], c.nbytes) == 0
    for p in ptr:
        L.xgb_free(p)
    assert L.xgb_gemm_tc_status() == 0
    bound = 8 * 2.0 ** -49 * k * np.abs(a).max(1)[:, None] * np.abs(b).max(0)[None, :]
    assert np.all(np.abs(c.T - a @ b) <= bound)
    return best * 1e3


@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 300001), (4, 4, 100000), (33, 65, 20011), (130, 3, 16400), (5, 7, 8176), (5, 7, 8177)])
def test_long_k(m, n, k, ta, tb):
    product(m, n, k, ta, tb, np.random.default_rng(m + k))


def test_time():
    assert product(4, 4, 100000, 0, 0, np.random.default_rng(0)) <= 0.45
