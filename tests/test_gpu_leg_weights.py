"""Bond weights on the legs of a site tensor (one kernel over its fusion-tree pairs) against the oracle, which
contracts them one after the other: simple-update steps on abelian, fermionic and SU(2) site tensors, with uneven
degeneracies and sub-blocks of more than 256 entries.  After a step G and the site tensors are compared to the 1e-8
that SVD-based updates are compared to elsewhere."""
import numpy as np
import pytest

import oracle
from oracle.basis import Qbasis
from oracle.ctm import IPEPS
from oracle.simple_update import SimpleUpdate as OSU
from oracle.simple_update import gate
from oracle.tensor import Tensor as OTensor

from helpers import assert_same, to_native

pytestmark = pytest.mark.gpu

PATTERN = [[0, 1], [1, 0]]


@pytest.mark.parametrize("symname,native,aux_p,phys_p,D", [
    ("u1", "U1", [(-1, 1), (0, 3), (1, 2)], [(-1, 1), (1, 1)], 5),
    ("u1", "U1", [(0, 5)], [(0, 2)], 5),
    ("fz2", "fZ2", [(0, 1), (1, 3)], [(0, 1), (1, 1)], 4),
    ("fu1", "fU1", [(-1, 2), (0, 1), (1, 1)], [(0, 1), (1, 1)], 4),
    ("su2", "SU2", [(1, 2), (2, 1), (3, 1)], [(2, 1)], 4),
])
def test_weights_match_contractions(symname, native, aux_p, phys_p, D):
    from xped_gb300 import Basis, SimpleUpdate, ensure_device
    ensure_device(0)
    s = oracle.make_symmetry(symname)
    oaux, ophys = Qbasis.from_pairs(s, aux_p), Qbasis.from_pairs(s, phys_p)
    naux, nphys = Basis.from_pairs(native, aux_p), Basis.from_pairs(native, phys_p)
    rng = np.random.default_rng(17)
    oG = [IPEPS(s, oaux, ophys).set_random(rng).A for _ in range(2)]
    nG = [to_native(g, [naux, naux], [naux, naux, nphys]) for g in oG]
    H = OTensor(s, [ophys, ophys], [ophys, ophys])
    for i, b in enumerate(H.blocks):
        r = rng.standard_normal(b.shape)
        H.blocks[i] = r + r.T
    oU = gate(H, 0.05)
    nU = to_native(oU, [nphys, nphys], [nphys, nphys])
    osu, nsu = OSU(PATTERN, oG, D), SimpleUpdate(PATTERN, nG, D)
    for i in range(2):
        assert_same(nsu.get("A", i), osu.site_tensor(i), 1e-12, 1e-14)
    osu.step_h(0, 0, oU)
    nsu.step_h(0, 0, nU)
    osu.step_v(1, 0, oU)
    nsu.step_v(1, 0, nU)
    for i in range(2):
        assert_same(nsu.get("G", i), osu.G[i], 1e-8, 1e-12)
        assert_same(nsu.get("A", i), osu.site_tensor(i), 1e-8, 1e-12)
