"""Powers of two on the columns of a block are exact, so they change nothing but the exponents: QR of a block whose
trailing columns (no pivots of their own) lie hundreds of binary orders from the leading ones must give the bits of the
unscaled problem."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(name, desc, sizes, a):
    """One block through xgb_batched_<name>: outputs of the given numbers of doubles."""
    from xped_gb300 import ensure_device, lib
    from xped_gb300._lib import last_error
    ensure_device(0)
    L = lib()
    work = getattr(L, f"xgb_{name}_workspace_bytes")(1, desc)
    ptr = []
    for nbytes in (a.nbytes, *(8 * n for n in sizes), work):
        p = C.c_void_p()
        assert L.xgb_malloc(C.byref(p), nbytes) == 0
        ptr.append(p)
    assert L.xgb_memcpy_h2d(ptr[0], a.ctypes.data, a.nbytes) == 0
    assert getattr(L, f"xgb_batched_{name}")(1, desc, *ptr, None) == 0, last_error()
    out = []
    for n, p in zip(sizes, ptr[1:]):
        x = np.empty(n)
        assert L.xgb_memcpy_d2h(x.ctypes.data, p, x.nbytes) == 0
        out.append(x)
    for p in ptr:
        L.xgb_free(p)
    return out


@pytest.mark.parametrize("m,n", [(8, 14), (60, 200)])
@pytest.mark.parametrize("lead,trail", [(0, 900), (0, -900), (460, 600), (-460, -620), (-490, 540), (490, -540), (20, 940)])
def test_qr_with_trailing_columns_of_another_scale(m, n, lead, trail):
    from xped_gb300._lib import QrDesc
    d = (QrDesc * 1)(QrDesc(m=m, n=n, q_cols=m, r_rows=m))
    a = np.random.default_rng(m).standard_normal((n, m))  # column-major
    e = np.where(np.arange(n) < m, lead, trail)
    q0, r0 = run("qr", d, (m * m, m * n), a)
    q1, r1 = run("qr", d, (m * m, m * n), np.ldexp(a, e[:, None]))
    assert np.array_equal(q0, q1)
    assert np.array_equal(np.ldexp(r0.reshape(n, m), e[:, None]), r1.reshape(n, m))
