"""Batched Householder QR (xgb_batched_qr) against LAPACK at the sizes where its form changes (one CTA, clusters
of 2 to 8, the columns in global memory), square, tall and wide, with zero columns and zero blocks: Q and R of
generic blocks to 1e-11 (the signs are dlarfg's), orthonormal Q and A = Q R to 50 max(m, n) eps for all."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.2204460492503131e-16
SHAPES = [(1, 1), (1, 6), (5, 9), (9, 5), (16, 16), (17, 17), (33, 32), (40, 33), (64, 128), (129, 128), (300, 65),
          (31, 200), (700, 130), (7040, 3), (7041, 2), (420, 500)]


@pytest.mark.parametrize("kind", ["gaussian", "zero_columns", "zero"])
def test_batched_qr_matches_lapack(kind):
    from xped_gb300 import ensure_device, lib
    from xped_gb300._lib import QrDesc, last_error
    ensure_device(0)
    L = lib()
    rng = np.random.default_rng(11)
    mats, descs, a, q, r = [], [], 0, 0, 0
    for m, n in SHAPES:
        k = min(m, n)
        A = np.zeros((m, n)) if kind == "zero" else rng.standard_normal((m, n))
        if kind == "zero_columns":
            A[:, ::3] = 0.0
        mats.append(A)
        descs.append(QrDesc(m, n, a, q, k, r, k))
        a, q, r = a + m * n, q + m * k, r + k * n
    arr = (QrDesc * len(descs))(*descs)
    flat = np.concatenate([x.ravel(order="F") for x in mats])
    ptr = []
    for nbytes in (flat.nbytes, 8 * q, 8 * r, L.xgb_qr_workspace_bytes(len(descs), arr)):
        p = C.c_void_p()
        assert L.xgb_malloc(C.byref(p), nbytes) == 0
        ptr.append(p)
    assert L.xgb_memcpy_h2d(ptr[0], flat.ctypes.data, flat.nbytes) == 0
    assert L.xgb_batched_qr(len(descs), arr, *ptr, None) == 0, last_error()
    assert L.xgb_synchronize() == 0
    hq, hr = np.empty(q), np.empty(r)
    assert L.xgb_memcpy_d2h(hq.ctypes.data, ptr[1], hq.nbytes) == 0
    assert L.xgb_memcpy_d2h(hr.ctypes.data, ptr[2], hr.nbytes) == 0
    for p in ptr:
        L.xgb_free(p)
    for A, d in zip(mats, descs):
        m, n = A.shape
        k, tol = min(m, n), 50 * max(m, n) * EPS
        Q = hq[d.q_off:d.q_off + m * k].reshape((m, k), order="F")
        R = hr[d.r_off:d.r_off + k * n].reshape((k, n), order="F")
        assert np.abs(np.tril(R[:, :k], -1)).max(initial=0) == 0.0
        assert np.abs(Q.T @ Q - np.eye(k)).max() <= tol, (m, n)
        assert np.linalg.norm(Q @ R - A) <= tol * max(np.linalg.norm(A), 1e-300), (m, n)
        if kind == "gaussian":
            refq, refr = np.linalg.qr(A)
            assert np.abs(Q - refq).max() <= 1e-11 and np.abs(R - refr).max() <= 1e-11 * np.abs(refr).max(), (m, n)
