"""FP64 grouped GEMM at the edges of its tiles: every extent around the 8 x 4 outputs of a warp, the 16-wide
sub-blocks and the tiles of 16, 32 and 64, both orientations of the operands, with and without split-K, alpha and
beta.  Each entry is a sum of k products in some order, then alpha and beta: the error is at most
(k + 8) eps (|alpha| |A| |B| + |beta C|) entrywise."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.2204460492503131e-16
EXTENTS = [(1, 1, 1), (4, 8, 3), (5, 9, 16), (8, 4, 17), (9, 5, 15), (15, 16, 33), (16, 15, 40), (17, 33, 64),
           (24, 20, 1), (31, 36, 31), (33, 17, 130), (40, 52, 70), (48, 49, 16), (63, 65, 200), (64, 64, 64),
           (65, 63, 129), (72, 12, 300), (100, 130, 90), (3, 150, 257), (150, 2, 300)]


@pytest.mark.parametrize("tile", [16, 32, 64])
@pytest.mark.parametrize("split,alpha,beta", [(0, 1.0, 0.0), (4, -0.75, 0.5)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_grouped_gemm_edges(tile, split, alpha, beta, ta, tb):
    from xped_gb300 import ensure_device, lib
    from xped_gb300._lib import GemmDesc, last_error
    ensure_device(0)
    L = lib()
    rng = np.random.default_rng(tile + 7 * split + ta + 2 * tb)
    descs, mats, a, b, c = [], [], 0, 0, 0
    for m, n, k in EXTENTS:
        A, B, D = (rng.standard_normal(s) for s in (((k, m) if ta else (m, k)), ((n, k) if tb else (k, n)), (m, n)))
        descs.append(GemmDesc(m, n, k, a, A.shape[0], b, B.shape[0], c, m, ta, tb))
        mats.append((A, B, D))
        a, b, c = a + m * k, b + n * k, c + m * n
    arr = (GemmDesc * len(descs))(*descs)
    bufs = [np.concatenate([x[i].ravel(order="F") for x in mats]) for i in range(3)]
    ptr = []
    for h in bufs:
        p = C.c_void_p()
        assert L.xgb_malloc(C.byref(p), h.nbytes) == 0
        assert L.xgb_memcpy_h2d(p, h.ctypes.data, h.nbytes) == 0
        ptr.append(p)
    assert L.xgb_grouped_gemm_f64_config(tile, split, len(descs), arr, *ptr, alpha, beta, None) == 0, last_error()
    out = np.empty_like(bufs[2])
    assert L.xgb_memcpy_d2h(out.ctypes.data, ptr[2], out.nbytes) == 0
    for p in ptr:
        L.xgb_free(p)
    for (m, n, k), d, (A, B, D) in zip(EXTENTS, descs, mats):
        A, B = (A.T if ta else A), (B.T if tb else B)
        got = out[d.c_off:d.c_off + m * n].reshape((m, n), order="F")
        exact = alpha * (A.astype(np.longdouble) @ B.astype(np.longdouble)) + beta * D
        bound = (k + 8) * EPS * (abs(alpha) * (np.abs(A) @ np.abs(B)) + abs(beta * D))
        assert (np.abs(got - exact) <= bound).all(), (m, n, k)
