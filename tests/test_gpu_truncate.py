"""Global truncation (xgb_truncate) against a sequential restatement of cutoff_matrices
(src/Core/Tensor.cpp:523-633) with the tie rule of the oracle: sizes around the 1024-thread CTA and the
shared-memory capacity, exact ties, near ties, zeros, eps and PRESERVE_MULTIPLETS."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TIE = 1e-12


def reference(s, begin, deg, max_keep, eps, preserve):
    n = len(s)
    exact = sorted(range(n), key=lambda i: (-s[i], i))
    order, group = [], []
    for p, i in enumerate(exact):
        if p and s[exact[p - 1]] - s[i] > TIE * s[exact[p - 1]]:
            order += sorted(group)
            group = []
        group.append(i)
    order += sorted(group)
    lim = min(n, max_keep)
    kept = [i for i in order[:lim] if not (eps > 0 and s[i] < eps)]
    if preserve:
        for k in range(len(kept) - 1, 0, -1):
            a, b = s[kept[k - 1]], s[kept[k]]
            if 2 * (a - b) / (a + b) > 0.1:
                kept = kept[:k]
                break
    if not kept:
        kept = [0]
    sector = np.searchsorted(begin, np.arange(n), side="right") - 1
    keep = np.zeros(len(deg), np.int32)
    for i in kept:
        keep[sector[i]] += 1
    weight = sum(deg[sector[i]] * s[i] ** 2 for i in order[lim:])
    with np.errstate(all="ignore"):
        entropy = sum(-deg[sector[i]] * s[i] ** 2 * np.log(s[i] ** 2) for i in kept)
    return keep, weight, entropy


@pytest.mark.parametrize("total", [1, 2, 33, 1023, 1024, 1025, 2049, 8192, 8193])
@pytest.mark.parametrize("eps,preserve", [(0.0, 0), (1e-3, 0), (1e-3, 1)])
def test_truncate_matches_restatement(total, eps, preserve):
    from xped_gb300 import ensure_device, lib
    from xped_gb300._lib import last_error
    ensure_device(0)
    L = lib()
    rng = np.random.default_rng(total)
    cuts = np.sort(rng.integers(0, total + 1, size=3))
    begin = np.array([0, *cuts, total], np.int64)
    deg = np.array([1, 3, 2, 1], np.int32)
    s = np.exp(-8 * rng.random(total))
    if total > 30:  # exact ties across sectors, ties within the tolerance, zeros below a kept value
        s[total // 2] = s[3]
        s[total // 3] = s[7] * (1 + 3e-13)
        s[[5, total - 1]] = 1e-300
    ptr = []
    for nbytes in (8 * total, 4 * 4, 16):
        p = C.c_void_p()
        assert L.xgb_malloc(C.byref(p), nbytes) == 0
        ptr.append(p)
    assert L.xgb_memcpy_h2d(ptr[0], s.ctypes.data, s.nbytes) == 0
    for max_keep in sorted({1, max(total // 2, 1), total + 5}):
        rc = L.xgb_truncate(4, begin.ctypes.data_as(C.POINTER(C.c_int64)), deg.ctypes.data_as(C.POINTER(C.c_int32)),
                            ptr[0], max_keep, eps, preserve, ptr[1], ptr[2], None)
        assert rc == 0, last_error()
        assert L.xgb_synchronize() == 0
        keep, out2 = np.zeros(4, np.int32), np.zeros(2)
        assert L.xgb_memcpy_d2h(keep.ctypes.data, ptr[1], keep.nbytes) == 0
        assert L.xgb_memcpy_d2h(out2.ctypes.data, ptr[2], out2.nbytes) == 0
        ref_keep, weight, entropy = reference(s, begin, deg, max_keep, eps, preserve)
        assert keep.tolist() == ref_keep.tolist()
        assert abs(out2[0] - weight) <= 1e-12 * max(1.0, weight)
        # a kept value whose square underflows gives 0 * log(0) = NaN on both sides
        assert np.isnan([out2[1], entropy]).all() or abs(out2[1] - entropy) <= 1e-11 * max(1.0, abs(entropy))
    for p in ptr:
        L.xgb_free(p)
