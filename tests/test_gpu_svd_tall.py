"""Exact SVD of tall (or flat) blocks of few columns against LAPACK, to 50 max(m, n) eps as in test_gpu_svd_forms.py, and
the cycles that one of a single column may take on its SM."""
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
