"""Calls on a stream of the caller's while the library's own stream allocates and frees: the temporaries of such a call
(descriptor tables, the truncation workspace beyond 8192 values) belong to the caller's stream.  The caller's stream is
kept busy first, so that each call's kernel runs long after the call has returned and has released its temporaries."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_truncate import reference
from test_permute_planes import build, expected

pytestmark = pytest.mark.gpu

SHAPES = [[(5, 7, 3)] * 40, [(9, 4), (3, 8, 5)] * 25, [(2, 2, 2, 3)] * 60]


def test_temporaries_follow_the_callers_stream():
    import torch
    from xped_gb300 import ensure_device, lib
    from xped_gb300._lib import last_error
    ensure_device(0)
    L = lib()
    plans = [build(sh, 20 + i, 0, 2, 1) for i, sh in enumerate(SHAPES)]
    dev = [(torch.from_numpy(src).cuda(), torch.full((size,), -7.5, dtype=torch.float64, device="cuda"))
           for _, _, src, size in plans]
    rng = np.random.default_rng(4)
    total, deg = 20000, np.array([1, 2, 1], np.int32)
    begin = np.array([0, 7000, 15000, total], np.int64)
    s = np.exp(-8 * rng.random(total))
    values = torch.from_numpy(s).cuda()
    keep = torch.zeros(3, dtype=torch.int32, device="cuda")
    out2 = torch.zeros(2, dtype=torch.float64, device="cuda")
    own = [(torch.from_numpy(src).cuda(), torch.zeros(size, dtype=torch.float64, device="cuda"))
           for _, _, src, size in plans]
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    busy = torch.zeros(1 << 26, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for _ in range(60):  # some tens of milliseconds of copies
            busy.add_(1.0)
    for (tasks, cons, _, _), (src, dst) in zip(plans, dev):
        assert L.xgb_permute(len(tasks), tasks, len(cons), cons, src.data_ptr(), dst.data_ptr(), stream.cuda_stream) == 0, last_error()
    assert L.xgb_truncate(3, begin.ctypes.data_as(C.POINTER(C.c_int64)), deg.ctypes.data_as(C.POINTER(C.c_int32)),
                          values.data_ptr(), 9000, 1e-3, 0, keep.data_ptr(), out2.data_ptr(), stream.cuda_stream) == 0, last_error()
    for _ in range(50):  # the library's own stream meanwhile
        for (tasks, cons, _, _), (src, dst) in zip(reversed(plans), reversed(own)):
            assert L.xgb_permute(len(tasks), tasks, len(cons), cons, src.data_ptr(), dst.data_ptr(), None) == 0, last_error()
    assert L.xgb_synchronize() == 0
    stream.synchronize()
    for (tasks, cons, src, size), (_, dst), (_, mine) in zip(plans, dev, own):
        want = expected(tasks, cons, src, size)
        assert np.array_equal(dst.cpu().numpy(), want)
        touched = want != -7.5
        assert np.array_equal(mine.cpu().numpy()[touched], want[touched])
    ref_keep, weight, entropy = reference(s, begin, deg, 9000, 1e-3, 0)
    assert np.array_equal(keep.cpu().numpy(), ref_keep)
    np.testing.assert_allclose(out2.cpu().numpy(), [weight, entropy], rtol=1e-11)
