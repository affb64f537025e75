"""CholeskyQR of the randomized tSVD at the sketch widths where its factorisation changes form (one CTA, clusters of 4
and 8, global memory), around the 16-wide panels, with narrow blocks beside wide ones: the kept singular vectors are
orthonormal to CholeskyQR's bound 6 (m l + l (l + 1)) u per basis, and the kept singular values are LAPACK's to 1e-10 of
the largest (the discarded spectrum is 1e-7 of the kept one, and four iterations reduce its share by 1e-7 each)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 1.1102230246251565e-16
LISTS = [[1, 2, 15, 16, 17], [31, 32, 33, 5], [47, 48, 1, 30], [49, 16, 2], [63, 64, 17], [65, 48, 1],
         [127, 128, 33, 15], [129, 112, 20], [200, 161], [320, 305, 33], [321, 20]]


@pytest.mark.parametrize("widths", LISTS)
def test_sketch_bases_are_orthonormal(widths):
    from xped_gb300 import Basis, Tensor
    rng = np.random.default_rng(sum(widths))
    dims = [2 * w + 3 for w in widths]
    basis = Basis.from_pairs("U1", list(enumerate(dims)))
    t = Tensor.zeros([basis], [basis])
    blocks, exact = [], []
    keep = [max(1, w - 4) for w in widths]
    for m, k in zip(dims, keep):
        u, v = (np.linalg.qr(rng.standard_normal((m, m)))[0] for _ in range(2))
        s = np.concatenate([np.linspace(2.0, 1.0, k), 1e-7 * np.linspace(1.0, 0.5, m - k)])
        blocks.append((u * s) @ v.T)
        exact.append(s[:k])
    t.set_data(np.concatenate([b.ravel(order="F") for b in blocks]))
    Uq, S, Vt, *_ = t.tSVD_randomized(sum(keep), 1e-5, widths, 4, seed=3)
    assert S.sectors()[1] == keep
    Ub, Sb, Vb = Uq.blocks(), S.blocks(), Vt.blocks()
    for q, (m, w, k, e) in enumerate(zip(dims, widths, keep, exact)):
        u, s, v = Ub[q], Sb[q], Vb[q]
        bound = 3 * 6 * (m * w + w * (w + 1)) * U  # Q of A, Q of A^T, and the small factors
        assert np.abs(u.T @ u - np.eye(k)).max() <= bound
        assert np.abs(v @ v.T - np.eye(k)).max() <= bound
        assert np.abs(np.diag(s) - e).max() <= 1e-10 * 2.0
