"""Boxes of few node rows in y: tiles of 4 and 8 rows, alone and with remainders (GPU).

Row counts around what a tile of each height finishes (3, 7, 15 and one more), on both levels, with equal and unequal
spacing, planes staged by tensor copies and by cp.async, deep enough in z that a chunk holds several planes.  FP64
against the C oracle (1e-12 for one operator, 1e-10 for a cycle), FP32 against FP64 after one flexible-PCG iteration
(1.2e-4 of the largest step: 20 applies of 1e2 x 6e-8).
"""
import numpy as np
import pytest

from oracle.bindings import COracle
from hpcrack_b200.solver import Hierarchy
from cases import D, R, RU, U, load_random, rel

pytestmark = pytest.mark.gpu
MG = (3, 2, 1, 1, 1)


@pytest.mark.parametrize("roi", [(0, 0, 0), (1, 2, 0)], ids=["equal", "unequal"])
@pytest.mark.parametrize("ey", [1, 3, 4, 8, 9])  # finest 3, 7, 9, 17, 19 rows; coarse 2, 4, 5, 9, 10
def test_thin_box(ey, roi):
    enb = (60, ey, 40)
    orc = COracle(1, enb, roi=roi)

    def operators(h):
        load_random([h], 1, enb, seed=6)
        out = []
        h.internal_force(0, U, RU, 1e-5)
        out.append((1e-12, h.get(RU, 0)))
        for l in (0, 1):
            h.fld(l, D, R, 2.0)
            out.append((1e-12, h.get(R, l)))
            h.fd_h(l)
        h.phase_field(MG, 2.0, 1, 1.0, pf_tol=1e-30)
        h.u_entire(MG, 1e-5, 1.0, 1, 1.0, mech_tol=1e-30)
        return out + [(1e-10, h.get(D, 1)), (1e-10, h.get(U, 1))]

    want = operators(orc)
    orc.close()
    for tma in (True, False):
        steps = []
        with Hierarchy(1, enb, roi=roi) as h:
            h.set_tma_staging(tma)
            for i, ((tol, a), (_, b)) in enumerate(zip(operators(h), want)):
                assert rel(a, b) < tol, (tma, i)
            for mixed in (False, True):
                load_random([h], 1, enb, seed=8)
                h.dirichlet_bd(1, U, 0.5)
                u0 = h.get(U, 1)
                h.u_entire_fcg((12, 2, 2, 1, 1), 1e-5, 0.5, 1, 1.0, mech_tol=1e-30, mixed=mixed)
                steps.append(h.get(U, 1) - u0)
        assert np.abs(steps[1] - steps[0]).max() <= 1.2e-4 * np.abs(steps[0]).max(), tma
