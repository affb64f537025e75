"""A power of two on a block is exact: the SVD of a block far from one must give the bits of the unscaled one, with its
singular values scaled."""
import numpy as np
import pytest

from test_gpu_qr_scales import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(20, 20), (90, 70)])
@pytest.mark.parametrize("e", [260, 400, -260, -400])
def test_svd_far_from_one(m, n, e):
    from xped_gb300._lib import SvdDesc
    d = (SvdDesc * 1)(SvdDesc(m=m, n=n))
    a = np.random.default_rng(m).standard_normal((n, m))
    sizes = (m * n, n, n * n)
    u0, s0, v0 = run("svd", d, sizes, a)
    u1, s1, v1 = run("svd", d, sizes, np.ldexp(a, e))
    assert np.array_equal(np.ldexp(s0, e), s1)
    assert np.array_equal(u0, u1) and np.array_equal(v0, v1)
