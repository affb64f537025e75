"""Batched QR of so many blocks that they take fewer CTAs each, and of blocks with several columns to a warp: the bits of
each block's own call (which takes as many CTAs as it can), and against LAPACK to 50 max(m, n) eps."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.2204460492503131e-16
BATCHES = {
    "all_alike": [(60, 60)] * 60 + [(61, 59)] * 60,
    "wide": [(30, 500)] * 40 + [(1, 300), (2, 65), (31, 33)],
    "one_long_chain": [(40, 40)] * 150 + [(300, 128)],
    "long_chains": [(300, 128)] * 30 + [(129, 97)] * 10 + [(4, 4)] * 200,
    "alone": [(33, 700)],
}


def batched_qr(mats):
    from xped_gb300 import ensure_device, lib
    from xped_gb300._lib import QrDesc, last_error
    ensure_device(0)
    L = lib()
    descs, a, q, r = [], 0, 0, 0
    for x in mats:
        m, n = x.shape
        k = min(m, n)
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
    return [(hq[d.q_off:d.q_off + d.m * d.q_cols].reshape((d.m, d.q_cols), order="F"),
             hr[d.r_off:d.r_off + d.r_rows * d.n].reshape((d.r_rows, d.n), order="F")) for d in descs]


@pytest.mark.parametrize("name", sorted(BATCHES))
def test_crowded_batches(name):
    rng = np.random.default_rng(sorted(BATCHES).index(name))
    mats = [rng.standard_normal(s) for s in BATCHES[name]]
    together = batched_qr(mats)
    seen = {}
    for x, (q, r) in zip(mats, together):
        m, n = x.shape
        k, tol = min(m, n), 50 * max(m, n) * EPS
        assert np.abs(q.T @ q - np.eye(k)).max() <= tol, (m, n)
        assert np.linalg.norm(q @ r - x) <= tol * np.linalg.norm(x), (m, n)
        if seen.setdefault((m, n), 0) < 2:
            seen[m, n] += 1
            own_q, own_r = batched_qr([x])[0]
            assert np.array_equal(q, own_q) and np.array_equal(r, own_r), (m, n)


@pytest.mark.parametrize("shapes", [[(1, 1)], [(8, 4)] * 9, [(4, 4), (9, 3), (2, 4), (1, 4), (2, 1)],
                                    [(3128, 4), (4693, 1), (3, 2)], [(3129, 4)], [(4694, 1)]], ids=str)
def test_batches_of_one_launch(shapes):
    """Q formed beside R (blocks of at most four columns that fit) or, in a batch with a wider block, by its own kernel."""
    rng = np.random.default_rng(len(shapes))
    mats = [rng.standard_normal(s) for s in shapes]
    if len(mats) > 2:
        mats[1][:, 0] = 0.0
    wider = rng.standard_normal((20, 17))
    for x, (q, r), (q2, r2) in zip(mats, batched_qr(mats), batched_qr(mats + [wider])):
        m, n = x.shape
        k, tol = min(m, n), 50 * max(m, n) * EPS
        assert np.abs(q.T @ q - np.eye(k)).max() <= tol, (m, n)
        assert np.linalg.norm(q @ r - x) <= tol * np.linalg.norm(x), (m, n)
        assert np.array_equal(q, q2) and np.array_equal(r, r2), (m, n)
