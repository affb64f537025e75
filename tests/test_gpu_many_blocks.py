"""Batches of more blocks than a grid's second extent holds (65535): the last block, wide enough for the refinement
products and for more than one column group of Q, and a sample of the narrow ones before it, against LAPACK."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNT = 65540
EPS = 2.2204460492503131e-16


def device(L, nbytes):
    p = C.c_void_p()
    assert L.xgb_malloc(C.byref(p), max(nbytes, 8)) == 0
    return p


def test_svd_of_many_blocks():
    from xped_gb300 import ensure_device, lib
    from xped_gb300._lib import SvdDesc, last_error
    ensure_device(0)
    L = lib()
    sizes = [(2, 2)] * (COUNT - 1) + [(40, 30)]
    rng = np.random.default_rng(6)
    a = rng.standard_normal(sum(m * n for m, n in sizes))
    d = (SvdDesc * COUNT)()
    at = [0, 0, 0, 0]
    for x, (m, n) in zip(d, sizes):
        k = min(m, n)
        x.m, x.n, x.a_off, x.u_off, x.s_off, x.vt_off = m, n, *at
        at = [p + q for p, q in zip(at, (m * n, m * k, k, k * n))]
    A, U, S, V = (device(L, 8 * q) for q in at)
    W = device(L, L.xgb_svd_workspace_bytes(COUNT, d))
    assert L.xgb_memcpy_h2d(A, a.ctypes.data, a.nbytes) == 0
    assert L.xgb_batched_svd(COUNT, d, A, U, S, V, W, None) == 0, last_error()
    u, s, v = (np.empty(q) for q in at[1:])
    for x, p in ((u, U), (s, S), (v, V)):
        assert L.xgb_memcpy_d2h(x.ctypes.data, p, x.nbytes) == 0
    for p in (A, U, S, V, W):
        L.xgb_free(p)
    for i in [0, 1, 65534, 65535, 65536, COUNT - 2, COUNT - 1]:
        x, (m, n) = d[i], sizes[i]
        k = min(m, n)
        blk = a[x.a_off:x.a_off + m * n].reshape(n, m).T
        ub, vb = u[x.u_off:x.u_off + m * k].reshape(k, m).T, v[x.vt_off:x.vt_off + k * n].reshape(n, k).T
        sb = s[x.s_off:x.s_off + k]
        tol = 50 * max(m, n) * EPS * np.linalg.norm(blk)
        assert np.abs(sb - np.linalg.svd(blk, compute_uv=False)).max() <= tol
        assert np.abs((ub * sb) @ vb - blk).max() <= tol


def test_qr_of_many_blocks():
    from xped_gb300 import ensure_device, lib
    from xped_gb300._lib import QrDesc, last_error
    ensure_device(0)
    L = lib()
    sizes = [(3, 2)] * (COUNT - 1) + [(40, 30)]
    rng = np.random.default_rng(7)
    a = rng.standard_normal(sum(m * n for m, n in sizes))
    d = (QrDesc * COUNT)()
    at = [0, 0, 0]
    for x, (m, n) in zip(d, sizes):
        k = min(m, n)
        x.m, x.n, x.a_off, x.q_off, x.r_off, x.q_cols, x.r_rows = m, n, *at, k, k
        at = [p + q for p, q in zip(at, (m * n, m * k, k * n))]
    A, Q, R = (device(L, 8 * q) for q in at)
    W = device(L, L.xgb_qr_workspace_bytes(COUNT, d))
    assert L.xgb_memcpy_h2d(A, a.ctypes.data, a.nbytes) == 0
    assert L.xgb_batched_qr(COUNT, d, A, Q, R, W, None) == 0, last_error()
    q, r = (np.empty(x) for x in at[1:])
    for x, p in ((q, Q), (r, R)):
        assert L.xgb_memcpy_d2h(x.ctypes.data, p, x.nbytes) == 0
    for p in (A, Q, R, W):
        L.xgb_free(p)
    for i in [0, 1, 65534, 65535, 65536, COUNT - 2, COUNT - 1]:
        x, (m, n) = d[i], sizes[i]
        k = min(m, n)
        blk = a[x.a_off:x.a_off + m * n].reshape(n, m).T
        qb, rb = q[x.q_off:x.q_off + m * k].reshape(k, m).T, r[x.r_off:x.r_off + k * n].reshape(n, k).T
        tol = 50 * max(m, n) * EPS * np.linalg.norm(blk)
        assert np.abs(qb @ rb - blk).max() <= tol
        assert np.abs(qb.T @ qb - np.eye(k)).max() <= 50 * max(m, n) * EPS
