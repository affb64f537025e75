"""Exact SVD of tall (or flat) blocks of few columns against LAPACK, to 50 max(m, n) eps as in test_gpu_svd_forms.py, the
cycles that one of a single column may take on its SM, and the share of a very tall one's time that is not its FP32
sweeps."""
import time

import numpy as np
import pytest

from test_gpu_svd_wide import block, check, decompose

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["gaussian", "graded12", "pairs", "deficient", "zero"])
@pytest.mark.parametrize("m,n", [(5000, 1), (1, 255), (256, 1), (257, 3), (870, 16), (9, 1400), (560, 24)])
def test_thin_blocks_of_one_cta(m, n, kind):
    a = block(m, n, kind, np.random.default_rng(m + n))
    check(a, *decompose(a)[:3])


def test_a_column_does_not_wait_for_one_thread():
    a = np.random.default_rng(1).standard_normal((5000, 1))
    stats = decompose(a)[3]
    assert stats[4] <= 100, stats  # cycles / 1024 of the refinement: 64 for every row is 320 of them, an iteration


@pytest.mark.parametrize("kind", ["gaussian", "graded12", "pairs", "deficient", "zero"])
@pytest.mark.parametrize("m,n", [(20000, 1), (60000, 2), (40000, 3), (3, 9000), (20000, 9), (8191, 17), (8192, 33), (5000, 130),
                                 (4096, 300), (4095, 60)])
def test_tall_blocks_of_many_ctas(m, n, kind):
    a = block(m, n, kind, np.random.default_rng(m + n))
    check(a, *decompose(a)[:3])


def test_the_gram_products_of_a_tall_block_use_all_sms():
    a = np.random.default_rng(2).standard_normal((400000, 2))
    sweeps = decompose(a)[3][2] * 1024 / 1.9e9  # seconds of the FP32 sweeps on CTA 0's SM
    from xped_gb300 import lib
    svd, times = lib().xgb_batched_svd, []

    def timed(*args):
        lib().xgb_synchronize()
        t0 = time.perf_counter()
        rc = svd(*args)
        lib().xgb_synchronize()
        times.append(time.perf_counter() - t0)
        return rc

    lib().xgb_batched_svd = timed
    try:
        decompose(a)
    finally:
        lib().xgb_batched_svd = svd
    assert times[0] <= 2.5 * sweeps + 2e-3, (times[0], sweeps)
