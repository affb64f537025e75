"""Gather-permute by planes (xgb_permute): its launch plan walked on the host, and the kernel itself, against a sum of
strided numpy views.  Shapes sit at the edges of chunks, tiles and lane groups; legs chain or not, stand apart in
wider parents, have extent 1; one to three sources per sub-block, coefficients +-1 and others.  Sources are small
whole numbers and coefficients multiples of 1/8, so every sum is exact in any order and results must be equal."""
import ctypes as C
import itertools

import numpy as np
import pytest

# extents of the output sub-block, leg 0 fastest
SHAPES = [(), (1,), (5,), (4100,), (1, 3, 1), (3, 3), (31, 33), (32, 32), (33, 65), (4, 16), (5, 300), (300, 5),
          (2049, 2), (7, 1, 9), (2, 3, 2, 2), (17, 6, 19), (40, 30, 20), (3, 1, 5, 4, 2), (2, 2, 2, 2, 2, 2, 2, 3),
          (4, 3, 5, 2, 3, 2, 2)]


def strides(extents, order, pad):
    """element strides of legs laid out in `order` (first is fastest) inside a parent padded by `pad` per leg"""
    st, step = [0] * len(extents), 1
    for leg in order:
        st[leg] = step
        step *= extents[leg] + pad
    return st, max(step, 1)


def build(shapes, seed, pad, sources, spread=1):
    from xped_gb300._lib import PermContrib, PermTask
    rng = np.random.default_rng(seed)
    tasks, cons, d_at, s_at = [], [], 3, 2
    for dims in shapes:
        n = len(dims)
        dst, dn = strides(dims, range(n), pad if n > 1 else 0)
        t = PermTask(dst_base=d_at, nelem=int(np.prod(dims, dtype=np.int64)), rank=n, n_contrib=sources,
                     contrib0=len(cons))
        for k in range(n):
            t.dims[k], t.dst_stride[k] = dims[k], dst[k]
        order = list(rng.permutation(n))
        for c in range(sources):
            src, sn = strides(dims, order if c < 2 or sources > 3 else list(rng.permutation(n)), pad)
            p = PermContrib(src_base=s_at, coeff=[1.0, -1.0, 0.375][(c + len(tasks)) % 3])
            for k in range(n):
                p.src_stride[k] = src[k] * spread
            s_at += sn * spread
            cons.append(p)
        d_at += dn
        tasks.append(t)
    src = rng.integers(-99, 100, s_at).astype(np.float64)
    return (PermTask * len(tasks))(*tasks), (PermContrib * len(cons))(*cons), src, d_at


def expected(tasks, cons, src, size):
    out = np.full(size, -7.5)
    for t in tasks:
        dims = list(t.dims[:t.rank])
        view = lambda buf, base, st: np.lib.stride_tricks.as_strided(buf[base:], dims, [8 * x for x in st[:t.rank]])
        acc = np.zeros(dims)
        for c in cons[t.contrib0:t.contrib0 + t.n_contrib]:
            acc = acc + c.coeff * view(src, c.src_base, c.src_stride)
        view(out, t.dst_base, t.dst_stride)[...] = acc
    return out


CASES = ([(SHAPES, seed, pad, sources, 1) for seed, pad, sources in itertools.product(range(3), (0, 2), (0, 1, 2, 3))] +
         [([s], 5, 0, 1, 1) for s in SHAPES] +
         [([(3, 3, 2, 2)] * 1500, 6, 0, 1, 1),        # more tasks than the prefix sums held in shared memory
          ([(3, 5)], 8, 0, 1100, 1), ([(8, 9)] * 3, 9, 1, 300, 1),   # more sources than a batch has slots for
          ([(4, 3)], 7, 0, 1, 5_000_000),             # source offsets that need 64 bits in the plan
          ([(1030, 2050), (2050, 1025)], 10, 0, 1, 1)])  # transposed tiles of more than 4 M elements


@pytest.mark.parametrize("case", range(len(CASES)))
def test_host_walk_matches_numpy(case):
    from xped_gb300 import lib
    tasks, cons, src, size = build(*CASES[case])
    out, form = np.full(size, -7.5), C.c_int(-1)
    assert lib().xgb_permute_walk_host(len(tasks), tasks, len(cons), cons, src.ctypes.data, out.ctypes.data,
                                       C.byref(form)) == 0
    assert form.value in (0, 1)
    assert np.array_equal(out, expected(tasks, cons, src, size))


def test_both_forms_are_covered():
    from xped_gb300 import lib
    seen = set()
    for case in CASES[:-3]:
        tasks, cons, src, size = build(*case)
        out, form = np.zeros(size), C.c_int(-1)
        assert lib().xgb_permute_walk_host(len(tasks), tasks, len(cons), cons, src.ctypes.data, out.ctypes.data,
                                           C.byref(form)) == 0
        seen.add(form.value)
    assert seen == {0, 1}


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(CASES)))
def test_kernel_matches_numpy(case):
    from xped_gb300 import ensure_device, lib
    from xped_gb300._lib import last_error
    ensure_device(0)
    L = lib()
    tasks, cons, src, size = build(*CASES[case])
    ptr = []
    for nbytes in (src.nbytes, 8 * size):
        p = C.c_void_p()
        assert L.xgb_malloc(C.byref(p), nbytes) == 0
        ptr.append(p)
    out = np.full(size, -7.5)
    assert L.xgb_memcpy_h2d(ptr[0], src.ctypes.data, src.nbytes) == 0
    assert L.xgb_memcpy_h2d(ptr[1], out.ctypes.data, out.nbytes) == 0
    assert L.xgb_permute(len(tasks), tasks, len(cons), cons, ptr[0], ptr[1], None) == 0, last_error()
    assert L.xgb_memcpy_d2h(out.ctypes.data, ptr[1], out.nbytes) == 0
    for p in ptr:
        L.xgb_free(p)
    assert np.array_equal(out, expected(tasks, cons, src, size))
