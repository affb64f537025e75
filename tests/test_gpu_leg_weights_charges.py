"""Bond weights that carry fewer charges than the leg they act on.  In a unit cell whose sites have more than one right
neighbour, a step on one of the bonds truncates the weight that the other neighbours' legs meet as well; their tensors
lose the sectors that only the dropped charges reach, as when the weights are contracted (the oracle)."""
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

PATTERN = [[0, 1], [2, 0]]


@pytest.mark.parametrize("D", [1, 2])
@pytest.mark.parametrize("symname,native", [("u1", "U1"), ("fu1", "fU1")])
def test_a_weight_may_lack_charges_of_its_leg(symname, native, D):
    from xped_gb300 import Basis, SimpleUpdate, ensure_device
    ensure_device(0)
    aux, phys = [(-1, 1), (0, 1), (1, 1)], [(-1, 1), (1, 1)]
    s = oracle.make_symmetry(symname)
    oaux, ophys = Qbasis.from_pairs(s, aux), Qbasis.from_pairs(s, phys)
    naux, nphys = Basis.from_pairs(native, aux), Basis.from_pairs(native, phys)
    rng = np.random.default_rng(23)
    oG = [IPEPS(s, oaux, ophys).set_random(rng).A for _ in range(3)]
    nG = [to_native(g, [naux, naux], [naux, naux, nphys]) for g in oG]
    H = OTensor(s, [ophys, ophys], [ophys, ophys])
    for i, b in enumerate(H.blocks):
        r = rng.standard_normal(b.shape)
        H.blocks[i] = r + r.T
    oU = gate(H, 0.05)
    nU = to_native(oU, [nphys, nphys], [nphys, nphys])
    osu, nsu = OSU(PATTERN, oG, D), SimpleUpdate(PATTERN, nG, D)
    osu.step_h(0, 0, oU)
    nsu.step_h(0, 0, nU)
    for i in range(3):
        assert_same(nsu.get("A", i), osu.site_tensor(i), 1e-8, 1e-12)
