"""Boxes so wide and thin that one plane holds more tiles than the usual reduction buffer has places for (GPU).

A tile kernel launches one block per tile and z chunk and every block leaves its partial sums, so the context's
buffer has to hold a plane's tiles whatever the box.  Against the C oracle, with the bars of the tile tests: 1e-12 for
one operator, 1e-10 for a cycle of a few smoother iterations.
"""
import pytest

from oracle.bindings import COracle
from hpcrack_b200.solver import FD, Hierarchy, U
from cases import D, R, load_random, rel

pytestmark = pytest.mark.gpu


def _pair(enb, seed):
    impls = Hierarchy(1, enb), COracle(1, enb)
    load_random(impls, 1, enb, seed=seed)
    return impls


def test_mechanical_solve():
    gpu, orc = _pair((512, 432, 1), 3)  # finest 1025 x 865 x 3: 69 x 124 = 8556 FP64 tiles of 15 x 7 nodes
    for impl in (gpu, orc):
        impl.u_entire((2, 1, 1, 1, 1), 1e-5, 1.0, 1, 1.0, mech_tol=1e-30)
    assert rel(gpu.get(U, 1), orc.get(U, 1)) < 1e-10
    gpu.close()
    orc.close()


def test_phase_field_operator():
    gpu, orc = _pair((680, 681, 1), 4)  # finest 1361 x 1363 x 3: 91 x 91 = 8281 tiles of 15 x 15 nodes
    for impl in (gpu, orc):
        impl.fld(1, D, R, 2.0)
    assert rel(gpu.get(R, 1), orc.get(R, 1)) < 1e-12
    gpu.close()
    orc.close()


def test_sums_of_many_blocks():
    gpu, orc = _pair((366, 364, 1), 5)  # finest 733 x 729 x 3: 2401 tiles, whose sums a kernel of its own combines
    for impl in (gpu, orc):
        impl.set(FD, 1, impl.get(D, 1))
    n0 = gpu.launch_count()
    fd = [impl.pcg_d(1, 2.0, 2, 1, 1.0)[1] for impl in (gpu, orc)]
    assert gpu.launch_count() - n0 == 3 + 2 + 2 * 4  # the preconditioner; residual and its sums; direction, apply, sums, update
    assert abs(fd[0] - fd[1]) <= 1e-12 * fd[1]
    for f in (D, R):
        assert rel(gpu.get(f, 1), orc.get(f, 1)) < 1e-10, f
    gpu.close()
    orc.close()
