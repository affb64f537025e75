"""xgb_truncate on values that its order treats apart: zeros of both signs (equal, kept by index), against the restatement
of test_gpu_truncate.py, and NaN (below every number), for which the kept counts still have to add up."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_truncate import reference

pytestmark = pytest.mark.gpu


def truncate(s, begin, deg, max_keep, eps=0.0):
    from xped_gb300 import ensure_device, lib
    from xped_gb300._lib import last_error
    ensure_device(0)
    L = lib()
    keep, out2, ptr = np.zeros(len(deg), np.int32), np.zeros(2), []
    for x in (s, keep, out2):
        p = C.c_void_p()
        assert L.xgb_malloc(C.byref(p), x.nbytes) == 0
        assert L.xgb_memcpy_h2d(p, x.ctypes.data, x.nbytes) == 0
        ptr.append(p)
    assert L.xgb_truncate(len(deg), begin.ctypes.data_as(C.POINTER(C.c_int64)), deg.ctypes.data_as(C.POINTER(C.c_int32)),
                          ptr[0], max_keep, eps, 0, ptr[1], ptr[2], None) == 0, last_error()
    assert L.xgb_memcpy_d2h(keep.ctypes.data, ptr[1], keep.nbytes) == 0
    assert L.xgb_memcpy_d2h(out2.ctypes.data, ptr[2], out2.nbytes) == 0
    for p in ptr:
        L.xgb_free(p)
    return keep, out2


@pytest.mark.parametrize("total", [3, 64, 1100, 9000])
def test_zeros_of_both_signs(total):
    rng = np.random.default_rng(total)
    begin, deg = np.array([0, total // 3, total // 2, total], np.int64), np.array([1, 2, 1], np.int32)
    s = rng.random(total)
    s[rng.random(total) < 0.5] = 0.0
    s[rng.random(total) < 0.2] = -0.0
    for max_keep in (1, total // 2, total - 1, total):
        for eps in (0.0, 1e-6):
            keep, out2 = truncate(s, begin, deg, max(max_keep, 1), eps)
            ref_keep, weight, _ = reference(s, begin, deg, max(max_keep, 1), eps, 0)
            assert keep.tolist() == ref_keep.tolist()
            assert abs(out2[0] - weight) <= 1e-12 * max(1.0, weight)


@pytest.mark.parametrize("total", [2, 40, 1100, 9000])
def test_nan(total):
    rng = np.random.default_rng(total)
    begin, deg = np.array([0, total // 3, total // 2, total], np.int64), np.array([1, 2, 1], np.int32)
    s = rng.random(total)
    s[rng.random(total) < 0.3] = np.nan
    s[0] = np.nan
    for max_keep in (1, total // 2, total):
        keep, _ = truncate(s, begin, deg, max(max_keep, 1))
        assert keep.sum() == max(max_keep, 1)
        assert np.all(keep >= 0) and np.all(keep <= np.diff(begin))
