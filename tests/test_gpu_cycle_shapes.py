"""One V- or W-cycle against the C oracle where the transfers and the handed-down residual can go wrong (GPU).

Odd and even coarse extents around a warp's 32 columns, one coarse plane pair up to several plane chunks,
coarse levels smoothed in one cluster and by the per-iteration kernels, gamma = 2 (the second coarse visit
forms its own residual), no pre-smoothing, and a spacing that differs per axis.  (A 2^3 coarse level is left
out: without a node at mid-width x is free to translate, and every implementation's iterates grow without
bound, the oracle's to 1e56.)  A cycle is a few dozen
smoother iterations on well-conditioned random moduli: 1e-10, as for every cycle.
"""
import pytest

from oracle.bindings import COracle
from hpcrack_b200.solver import Hierarchy, GE, KE, U
from cases import D, load_random, rel

pytestmark = pytest.mark.gpu

CASES = [  # max_level, element_nb, roi, (nu0, nu1, nu2, gamma, ncy)
    (1, (31, 4, 9), (0, 0, 0), (12, 3, 2, 1, 1)),
    (1, (32, 5, 3), (0, 0, 0), (12, 3, 2, 1, 1)),
    (2, (5, 16, 7), (0, 0, 0), (12, 2, 1, 2, 1)),
    (2, (13, 14, 15), (0, 0, 0), (12, 2, 2, 2, 1)),  # level 1 too large for a cluster
    (2, (6, 4, 5), (1, 0, 2), (12, 0, 3, 1, 1)),
]


@pytest.mark.parametrize("ml,enb,roi,mg", CASES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_cycle(ml, enb, roi, mg):
    gpu, orc = Hierarchy(ml, enb, roi=roi), COracle(ml, enb, roi=roi)
    load_random([gpu, orc], ml, enb, seed=11)
    for impl in (gpu, orc):
        impl.mp_all_element(1e-5)
        impl.vr_all_level(KE)
        impl.vr_all_level(GE)
        for l in range(ml + 1):
            impl.fd_h(l)
    fn = [impl.cycle_u(ml, mg, 1e-5, 0.7, 0, 0.0)[1] for impl in (gpu, orc)]
    assert abs(fn[0] - fn[1]) <= 1e-10 * abs(fn[1])
    assert rel(gpu.get(U, ml), orc.get(U, ml)) < 1e-10
    for impl in (gpu, orc):
        impl.cycle_d(ml, mg, 2.0, 0, 0.0)
    assert rel(gpu.get(D, ml), orc.get(D, ml)) < 1e-10
    gpu.close()
    orc.close()
