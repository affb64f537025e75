"""The launch tables of the bond weights: one entry per pair of fusion trees, whatever the degeneracies.  What the cached
plan holds is read from the device's memory pool; values are compared with the tensor itself (all weights are one
before the first step), on legs with more pairs than the kernel keeps in shared memory too."""
import ctypes as C
import gc
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

USED_CURRENT = 0x7  # cudaMemPoolAttrUsedMemCurrent


def pool_bytes():
    from xped_gb300 import lib
    from xped_gb300.build import CUDA_HOME
    rt = C.CDLL(str(CUDA_HOME / "lib64" / "libcudart.so"))
    gc.collect()
    lib().xgb_synchronize()
    pool, used = C.c_void_p(), C.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, USED_CURRENT, C.byref(used)) == 0
    return used.value


@pytest.mark.parametrize("aux,phys", [([(0, 24)], [(0, 2)]), ([(-1, 9), (0, 13), (1, 8)], [(-1, 1), (1, 1)]),
                                      ([(q, 2) for q in range(-4, 5)], [(-1, 1), (1, 1)])])
def test_tables_do_not_grow_with_the_degeneracies(aux, phys):
    from xped_gb300 import Basis, SimpleUpdate, Tensor, ensure_device
    ensure_device(0)
    a, p = Basis.from_pairs("U1", aux), Basis.from_pairs("U1", phys)
    rng = np.random.default_rng(3)
    sites = []
    for _ in range(2):
        t = Tensor.zeros([a, a], [a, a, p])
        t.set_data(rng.standard_normal(t.size))
        sites.append(t)
    su = SimpleUpdate([[0, 1], [1, 0]], sites, 4)
    pairs = sum(l + t == r + b + s for l, t, r, b, s in itertools.product(*[[q for q, _ in aux]] * 4, [q for q, _ in phys]))
    before = pool_bytes()
    x = su.get("A", 0)
    assert np.array_equal(x.data(), sites[0].data())
    del x
    assert pool_bytes() - before <= 256 * pairs + 65536
