"""Smoother updates that move two steps at a time, leave out what nobody reads, and start from a zero unknown (GPU).

pcg_u against the C oracle on a level above the cluster size for odd and even iteration counts (an odd count
ends with a single step), and the flexible-PCG solves - whose cycles start from zero, with and without
pre- and post-smoothing - on a context that has just run the other precision's solve: the direction arrays are
shared between the precisions, so whatever they hold outside the grid must not matter.  Same kernels, same
order: equal bit for bit to a fresh context.
"""
import numpy as np
import pytest

from oracle.bindings import COracle
from hpcrack_b200.solver import Hierarchy, RU, U
from cases import D, H, load_random, rel

pytestmark = pytest.mark.gpu
ENB = (13, 14, 15)  # two levels: 29 x 27 x 31 nodes at the finest, rows of 27 with padding


@pytest.mark.parametrize("nb", [0, 1, 2, 3, 6])
def test_pcg_u_iteration_counts(nb):
    gpu, orc = Hierarchy(1, ENB), COracle(1, ENB)
    load_random([gpu, orc], 1, ENB, seed=5)
    for impl in (gpu, orc):
        impl.pcg_u(1, 1e-5, 0.5, nb, 1, 1.0)
    for f in (U, RU):
        assert rel(gpu.get(f, 1), orc.get(f, 1)) < 1e-10, f
    gpu.close()
    orc.close()


@pytest.mark.parametrize("nu", [(4, 4), (3, 2), (0, 3), (1, 0)], ids=lambda v: f"{v[0]}-{v[1]}")
def test_solves_share_direction_arrays(nu):
    mg = (12, nu[0], nu[1], 1, 3)

    def solve(gpu, mixed):
        load_random([gpu], 1, ENB, seed=7)
        gpu.u_entire_fcg(mg, 1e-5, 0.5, 1, 1.0, mech_tol=1e-30, mixed=mixed)
        return gpu.get(U, 1).copy()

    both = Hierarchy(1, ENB)
    for mixed in (False, True, False, True):
        got = solve(both, mixed)
        fresh = Hierarchy(1, ENB)
        want = solve(fresh, mixed)
        assert np.isfinite(want).all()
        np.testing.assert_array_equal(got, want)
        fresh.close()
    both.close()
