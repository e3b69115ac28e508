"""Tile kernels on chunks of many planes: stages refilled, waits of both parities, planes finished in a row (GPU).

On 129 x 97 x 65 nodes a chunk of the finest level holds 17 to 33 planes and one of the 65 x 49 x 33 level 3 to 5, the
planes no multiple of the chunks.  FP64 against the C oracle with equal and unequal spacing, planes staged by tensor copies
and by cp.async: 1e-12 for one operator, 1e-10 for a cycle, as in the tests of the tiles' edges.

FP32 against FP64 (which the oracle checks): one iteration of the flexible PCG takes u by alpha z, z one V-cycle, the
same cycle in both precisions.  An apply is a few hundred products and sums (at most 1e2 x 6e-8 of its result), a
cycle chains about 20 applies and transfers on well-conditioned moduli: 20 x 6e-6, 1.2e-4 of the largest step, at every
node, so that a wrong value at one tile's edge shows.
"""
import numpy as np
import pytest

from oracle.bindings import COracle
from hpcrack_b200.solver import Hierarchy
from cases import D, R, RU, U, load_random, rel

pytestmark = pytest.mark.gpu
ML, ENB = 2, (32, 24, 16)
MG = (2, 1, 1, 1, 1)


def _operators(h):
    """Coarse mechanical and phase-field operators, a phase-field cycle, a mechanical cycle."""
    out = []
    h.internal_force(1, U, RU, 1e-5)
    out.append(("K", 1e-12, h.get(RU, 1)))
    for l in (1, 2):
        h.fld(l, D, R, 2.0)
        out.append((f"A{l}", 1e-12, h.get(R, l)))
    for l in range(ML + 1):
        h.fd_h(l)
    h.phase_field(MG, 2.0, 1, 1.0, pf_tol=1e-30)
    h.u_entire(MG, 1e-5, 1.0, 1, 1.0, mech_tol=1e-30)
    return out + [("d", 1e-10, h.get(D, ML)), ("u", 1e-10, h.get(U, ML))]


@pytest.mark.parametrize("roi", [(0, 0, 0), (1, 2, 0)], ids=["equal", "unequal"])
def test_marched_chunks(roi):
    orc = COracle(ML, ENB, roi=roi)
    load_random([orc], ML, ENB, seed=9)
    want = _operators(orc)
    orc.close()
    for tma in (True, False):
        with Hierarchy(ML, ENB, roi=roi) as gpu:
            gpu.set_tma_staging(tma)
            load_random([gpu], ML, ENB, seed=9)
            for (name, tol, a), (_, _, b) in zip(_operators(gpu), want):
                assert rel(a, b) < tol, (name, tma)


@pytest.mark.parametrize("fused", [True, False], ids=["cluster", "per-iteration"])
@pytest.mark.parametrize("tma", [True, False], ids=["tma", "cp.async"])
@pytest.mark.parametrize("ml,enb,roi", [(1, (8, 9, 7), (0, 0, 0)), (2, (4, 5, 3), (1, 2, 0)), (ML, ENB, (0, 0, 0)),
                                        (ML, ENB, (1, 2, 0))], ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_fp32_cycle(ml, enb, roi, tma, fused):
    steps = []
    for mixed in (False, True):
        with Hierarchy(ml, enb, roi=roi) as h:
            h.set_tma_staging(tma)
            h.set_fused_coarsest(fused)
            load_random([h], ml, enb, seed=8)
            h.dirichlet_bd(ml, U, 0.5)
            u0 = h.get(U, ml)
            h.u_entire_fcg((12, 2, 2, 1, 1), 1e-5, 0.5, 1, 1.0, mech_tol=1e-30, mixed=mixed)
            steps.append(h.get(U, ml) - u0)
    d64, d32 = steps
    assert np.abs(d64).max() > 0
    assert np.abs(d32 - d64).max() <= 1.2e-4 * np.abs(d64).max()
