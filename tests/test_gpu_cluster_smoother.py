"""The one-cluster smoothers of small levels against the C oracle's pcg_u and pcg_d (GPU).

Levels cut along each axis, with fewer planes than blocks, one and several planes a block, a block whose
share is larger than its neighbours', each block shape (1 to 1024 elements a block), and a spacing that
differs per axis.  A smoother call is 1 to 6 iterations whose step lengths are quotients of sums: the
rounding of a sum in another order (1e-15) times the conditioning of a few iterations, 1e-10 as for
every smoother.
"""
import pytest

from oracle.bindings import COracle
from hpcrack_b200.solver import Hierarchy, RU, U
from cases import D, R, load_random, rel

pytestmark = pytest.mark.gpu

GEOMS = [
    ((1, 1, 1), (0, 0, 0)),     # 2^3 nodes
    ((4, 3, 2), (0, 0, 0)),     # cut along x, 5 planes
    ((3, 15, 4), (0, 0, 0)),    # along y, 16 planes, one a block
    ((8, 8, 8), (0, 0, 0)),     # along z, 9 planes
    ((12, 12, 12), (0, 0, 0)),  # 13 planes of 169 nodes
    ((16, 16, 16), (0, 0, 0)),  # 17 planes: one block has two
    ((40, 8, 16), (0, 0, 0)),   # 41 planes along x, two or three a block
    ((6, 20, 5), (1, 2, 0)),    # h differs per axis
    ((24, 24, 24), (0, 0, 0)),  # too large for a cluster: the per-iteration kernels
]


@pytest.mark.parametrize("enb,roi", GEOMS, ids=lambda v: "x".join(map(str, v)))
def test_cluster_smoother(enb, roi):
    gpu, orc = Hierarchy(1, enb, roi=roi), COracle(1, enb, roi=roi)
    load_random([gpu, orc], 1, enb, seed=3)
    for nb, Ut in ((1, 1.0), (6, 0.5)):
        for impl in (gpu, orc):
            impl.pcg_u(0, 1e-5, Ut, nb, 1, 1.0)
        for f in (U, RU):
            assert rel(gpu.get(f, 0), orc.get(f, 0)) < 1e-10, (nb, f)
        for impl in (gpu, orc):
            impl.fd_h(0)
        fd = [impl.pcg_d(0, 2.0, nb, 1, 1.0)[1] for impl in (gpu, orc)]
        assert abs(fd[0] - fd[1]) <= 1e-12 * fd[1]
        for f in (D, R):
            assert rel(gpu.get(f, 0), orc.get(f, 0)) < 1e-10, (nb, f)
    gpu.close()
    orc.close()
