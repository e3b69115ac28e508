"""A context whose solve ran into NaN serves the next solve as a fresh one does (GPU).

Vectors are stored with padding slots at the end of each row; kernels that work on pairs of slots read and write
them, so whatever a solve leaves there must not reach a later one.  Same kernels, same order: equal bit for bit.
"""
import numpy as np
import pytest

from hpcrack_b200.solver import Hierarchy, FU, U
from cases import load_random

pytestmark = pytest.mark.gpu
ENB = (13, 14, 15)  # rows of 27 and 14 nodes: padding on both levels
MG = (12, 3, 2, 1, 2)


def _solve(h, form, t=1):
    if form == "fas":
        h.u_entire(MG, 1e-5, 0.5, t, 1.0, mech_tol=1e-30)
    else:
        h.u_entire_fcg(MG, 1e-5, 0.5, t, 1.0, mech_tol=1e-30, mixed=form == "mixed")
    return h.get(U, 1).copy()


@pytest.mark.parametrize("fused", [True, False], ids=["cluster", "per-iteration"])
@pytest.mark.parametrize("form", ["fas", "fcg", "mixed"])
def test_solve_after_nan(form, fused):
    with Hierarchy(1, ENB) as used, Hierarchy(1, ENB) as fresh:
        for h in (used, fresh):
            h.set_fused_coarsest(fused)
        load_random([used], 1, ENB, seed=5)
        bad = np.zeros((3, used.n(1)))
        bad[1, used.n(1) // 2] = np.nan
        used.set(FU, 1, bad)
        assert np.isnan(_solve(used, form, t=0)).any()  # t = 0: the cycle runs whatever the first residual is
        for h in (used, fresh):
            load_random([h], 1, ENB, seed=6)
        want = _solve(fresh, form)
        assert np.isfinite(want).all()
        np.testing.assert_array_equal(_solve(used, form), want)
