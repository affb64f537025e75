"""Exact SVD of blocks from 512 columns on: held by a cluster (to 640 columns; second pass and FP64 sweeps on a
cooperative grid above 512), or too large for one (QR with column pivoting, then Jacobi), on lane 0 and on a side lane.
Against LAPACK to 50 max(m, n) eps as in test_gpu_svd_forms.py.  A block that no cluster holds must converge in the
sweeps of a preconditioned Jacobi (11 to 14 measured over these spectra; without the factor 20 to 60)."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_svd_forms import EPS, haar, spectrum

pytestmark = pytest.mark.gpu


def block(m, n, kind, rng):
    k = min(m, n)
    if kind == "gaussian":
        return rng.standard_normal((m, n))
    i = np.arange(k)
    s = {"graded12": 10.0 ** (-12.0 * i / k), "pairs": 10.0 ** (-14.0 * (i // 2) / (k // 2 + 1))}.get(kind)
    return (haar(rng, m, k) * (spectrum(kind, k) if s is None else s)) @ haar(rng, n, k).T


def decompose(a, lane=0):
    """U, S, V^T and the sweep counts of one block through xgb_batched_svd."""
    from xped_gb300 import ensure_device, lib
    from xped_gb300._lib import LIB_PATH, SvdDesc, last_error
    ensure_device(0)
    L = lib()
    m, n = a.shape
    k = min(m, n)
    d = (SvdDesc * 1)(SvdDesc(m=m, n=n))
    ptr = []
    for nbytes in (8 * m * n, 8 * m * k, 8 * k, 8 * k * n, L.xgb_svd_workspace_bytes(1, d)):
        p = C.c_void_p()
        assert L.xgb_malloc(C.byref(p), nbytes) == 0
        ptr.append(p)
    flat = np.ascontiguousarray(a.T)
    assert L.xgb_memcpy_h2d(ptr[0], flat.ctypes.data, flat.nbytes) == 0
    scope = C.create_string_buffer(64)
    if lane:  # xgb::LaneScope: what run_pair puts around each of its two sides
        native = C.CDLL(str(LIB_PATH))
        native._ZN3xgb9LaneScopeC1Ei(scope, lane)
    try:
        assert L.xgb_batched_svd(1, d, *ptr[:4], ptr[4], None) == 0, last_error()
    finally:
        if lane:
            native._ZN3xgb9LaneScopeD1Ev(scope)
    stats = (C.c_int32 * 6)()
    L.xgb_svd_last_sweeps(stats, 6)
    u, s, v = np.empty((k, m)), np.empty(k), np.empty((n, k))
    for arr, p in ((u, ptr[1]), (s, ptr[2]), (v, ptr[3])):
        assert L.xgb_memcpy_d2h(arr.ctypes.data, p, arr.nbytes) == 0
    for p in ptr:
        L.xgb_free(p)
    return u.T, s, v.T, list(stats)


def check(a, u, s, v):
    tol = 50 * max(a.shape) * EPS
    ref = np.linalg.svd(a, compute_uv=False)
    top = max(ref[0], 1e-300)
    live = s > 1e-12 * top
    assert np.abs(s - ref).max() <= tol * top
    assert np.abs(u[:, live].T @ u[:, live] - np.eye(live.sum())).max(initial=0) <= max(tol, 1e-12)
    assert np.abs(v[live] @ v[live].T - np.eye(live.sum())).max(initial=0) <= max(tol, 1e-12)
    assert np.linalg.norm((u * s) @ v - a) <= tol * max(np.linalg.norm(a), 1e-300)


@pytest.mark.parametrize("kind", ["gaussian", "power", "graded12", "pairs", "degenerate", "deficient", "zero"])
@pytest.mark.parametrize("m,n", [(641, 641), (700, 700), (1024, 900), (700, 1400), (1300, 512)])
def test_blocks_that_no_cluster_holds(m, n, kind):
    a = block(m, n, kind, np.random.default_rng(m + n))
    u, s, v, stats = decompose(a)
    check(a, u, s, v)
    assert stats[0] + stats[1] <= 20, stats


@pytest.mark.parametrize("kind", ["gaussian", "power", "graded12", "pairs", "degenerate", "deficient", "zero"])
@pytest.mark.parametrize("m,n", [(512, 512), (513, 513), (640, 640), (530, 900)])
def test_blocks_that_a_cluster_holds(m, n, kind):
    a = block(m, n, kind, np.random.default_rng(m + n))
    check(a, *decompose(a)[:3])


@pytest.mark.parametrize("kind", ["gaussian", "graded12", "pairs"])
@pytest.mark.parametrize("m,n", [(400, 400), (600, 600), (660, 700), (1400, 520)])
def test_wide_blocks_on_a_side_lane(m, n, kind):
    a = block(m, n, kind, np.random.default_rng(m + n))
    check(a, *decompose(a, lane=1)[:3])
