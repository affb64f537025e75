"""The thin SVD of sector blocks at the sizes where its form changes (one CTA, clusters of 1 to 16 CTAs, the
cooperative grid; the register heights of the FP32 sweeps; tall and wide blocks), against LAPACK, for generic,
graded, degenerate, rank-deficient and zero spectra: singular values, orthonormal factors (columns above
1e-12 of the largest value) and the reconstruction, each to 50 max(m, n) eps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.2204460492503131e-16
SHAPES = [(1, 1), (1, 8), (24, 24), (24, 500), (25, 25), (32, 33), (64, 64), (65, 65), (128, 96), (129, 128),
          (160, 160), (161, 200), (257, 256), (321, 320), (12, 3000), (2500, 40), (513, 512), (641, 600)]


def haar(rng, m, k):
    return np.linalg.qr(rng.standard_normal((m, k)))[0]


def spectrum(kind, k):
    i = np.arange(k)
    return {"power": (i + 1.0) ** -2, "graded": 10.0 ** (-9.0 * i / k),
            "degenerate": np.repeat(np.linspace(1, 0.1, (k + 3) // 4), 4)[:k],
            "deficient": np.where(i < (k + 1) // 2, 1.0, 0.0), "zero": np.zeros(k)}[kind]


@pytest.mark.parametrize("kind", ["gaussian", "power", "graded", "degenerate", "deficient", "zero"])
def test_svd_forms_match_lapack(kind):
    from xped_gb300 import Basis, Tensor
    rng = np.random.default_rng(5)
    blocks = {}
    for q, (m, n) in enumerate(SHAPES):
        k = min(m, n)
        blocks[q] = (rng.standard_normal((m, n)) if kind == "gaussian"
                     else (haar(rng, m, k) * spectrum(kind, k)) @ haar(rng, n, k).T)
    R = Basis.from_pairs("U1", [(q, m) for q, (m, _) in enumerate(SHAPES)])
    Cb = Basis.from_pairs("U1", [(q, n) for q, (_, n) in enumerate(SHAPES)])
    t = Tensor.zeros([R], [Cb])
    t.set_blocks(blocks)
    U, S, V, *_ = t.tSVD(1 << 30, 0.0)
    U, S, V = U.blocks(), S.blocks(), V.blocks()
    for q, (m, n) in enumerate(SHAPES):
        tol = 50 * max(m, n) * EPS
        ref = np.linalg.svd(blocks[q], compute_uv=False)
        if q not in S:  # a zero tensor keeps one value
            assert kind == "zero"
            continue
        s, top = np.diag(S[q]), max(ref[0], 1e-300)
        live = s > 1e-12 * top
        assert np.abs(s - ref[:len(s)]).max() <= tol * top, (m, n)
        u, v = U[q][:, live], V[q][live]
        assert np.abs(u.T @ u - np.eye(u.shape[1])).max(initial=0) <= max(tol, 1e-12), (m, n)
        assert np.abs(v @ v.T - np.eye(v.shape[0])).max(initial=0) <= max(tol, 1e-12), (m, n)
        assert np.linalg.norm((U[q] * s) @ V[q] - blocks[q]) <= tol * max(np.linalg.norm(blocks[q]), 1e-300), (m, n)
