"""Permutes whose output begins with two short legs: the plane is spanned with the longest of the other legs instead.  The
plan walked on the host and the kernel against numpy (exact sums, as in test_permute_planes.py), and the time of such a
permute against that of a plain copy of as many elements."""
import ctypes as C
import time

import numpy as np
import pytest

from test_permute_planes import build, expected

SHAPES = [(2, 3, 500), (3, 2, 7, 90), (2, 2, 2, 1000), (5, 6, 40), (2, 15, 3, 3), (4, 7, 2, 2, 600), (2, 2, 2, 2, 2, 3),
          (3, 10, 33, 2), (1, 2, 3, 2049)]
CASES = [(SHAPES, seed, pad, sources) for seed in range(4) for pad, sources in ((0, 1), (2, 1), (0, 3))]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_host_walk(case):
    from xped_gb300 import lib
    tasks, cons, src, size = build(*CASES[case])
    out, form = np.full(size, -7.5), C.c_int(-1)
    assert lib().xgb_permute_walk_host(len(tasks), tasks, len(cons), cons, src.ctypes.data, out.ctypes.data,
                                       C.byref(form)) == 0
    assert np.array_equal(out, expected(tasks, cons, src, size))


def device(L, host):
    p = C.c_void_p()
    assert L.xgb_malloc(C.byref(p), host.nbytes) == 0
    assert L.xgb_memcpy_h2d(p, host.ctypes.data, host.nbytes) == 0
    return p


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(CASES)))
def test_kernel(case):
    from xped_gb300 import ensure_device, lib
    from xped_gb300._lib import last_error
    ensure_device(0)
    L = lib()
    tasks, cons, src, size = build(*CASES[case])
    out = np.full(size, -7.5)
    s, d = device(L, src), device(L, out)
    assert L.xgb_permute(len(tasks), tasks, len(cons), cons, s, d, None) == 0, last_error()
    assert L.xgb_memcpy_d2h(out.ctypes.data, d, out.nbytes) == 0
    L.xgb_free(s)
    L.xgb_free(d)
    assert np.array_equal(out, expected(tasks, cons, src, size))


@pytest.mark.gpu
def test_a_plane_of_six_does_not_cost_its_decoding():
    from xped_gb300 import ensure_device, lib
    from xped_gb300._lib import PermContrib, PermTask
    ensure_device(0)
    L = lib()
    n = 5_000_000
    x = np.arange(6.0 * n)
    s, d = device(L, x), device(L, np.zeros_like(x))

    def milliseconds(src_stride):
        t = (PermTask * 1)(PermTask(nelem=6 * n, rank=3, n_contrib=1))
        c = (PermContrib * 1)(PermContrib(coeff=1.0))
        for k, (dim, dst) in enumerate(((2, 1), (3, 2), (n, 6))):
            t[0].dims[k], t[0].dst_stride[k], c[0].src_stride[k] = dim, dst, src_stride[k]
        best = 1e9
        for _ in range(8):
            L.xgb_synchronize()
            t0 = time.perf_counter()
            assert L.xgb_permute(1, t, 1, c, s, d, None) == 0
            L.xgb_synchronize()
            best = min(best, time.perf_counter() - t0)
        return best * 1e3

    copy, moved = milliseconds((1, 2, 6)), milliseconds((1, 2 * n, 2))  # [2, n, 3] -> [2, 3, n]
    out = np.empty_like(x)
    assert L.xgb_memcpy_d2h(out.ctypes.data, d, out.nbytes) == 0
    L.xgb_free(s)
    L.xgb_free(d)
    assert np.array_equal(out.reshape(n, 3, 2), x.reshape(3, n, 2).transpose(1, 0, 2))
    assert moved <= 4 * copy, (moved, copy)
