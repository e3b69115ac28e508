"""The tile kernels of the mechanical and phase-field operators against the C oracle (GPU) where tiles end.

A tile finishes 15 node columns in x and 7 (mechanical FP64) or 15 in y: levels whose extents are a tile,
one node less and one node more, levels smaller than a tile, and a spacing that differs per axis.
Coarse levels run through Internal_Force (element-constant moduli); the finest level's kernel on
precomputed Gauss-point moduli runs inside a mechanical solve, here one V-cycle of u_entire with its
residual, smoother and reaction applies.  One apply is a sum of a few hundred products (1e-12, the
bar of every operator); a cycle of 3 + 1 smoother iterations on a fixed right-hand side multiplies
that by the iterations and the conditioning of the step lengths: 1e-10.
"""
import pytest

from oracle.bindings import COracle
from hpcrack_b200.solver import Hierarchy
from cases import D, FD, FU, R, RU, U, load_random, rel

pytestmark = pytest.mark.gpu

GEOMS = [
    (1, (14, 6, 5), (0, 0, 0)),    # coarse 15 x 7 x 6 (one tile), finest 29 x 13 x 11
    (1, (15, 7, 3), (0, 0, 0)),    # coarse 16 x 8 x 4 (one node into the next tile), finest 31 x 15 x 7
    (1, (13, 5, 2), (0, 0, 0)),    # coarse 14 x 6 x 3, finest 27 x 11 x 5
    (1, (1, 1, 1), (0, 0, 0)),     # one element, finest 3^3
    (2, (4, 2, 9), (0, 0, 0)),     # 5 x 3 x 10, 9 x 5 x 19, 17 x 9 x 37
    (1, (8, 7, 4), (1, 2, 0)),     # h differs per axis
]


@pytest.mark.parametrize("tma", [True, False], ids=["tma", "cp.async"])
@pytest.mark.parametrize("geom", GEOMS, ids=lambda g: f"L{g[0]}-{g[1][0]}x{g[1][1]}x{g[1][2]}-roi{g[2][0]}{g[2][1]}{g[2][2]}")
def test_tile_apply(geom, tma):
    ml, enb, roi = geom
    gpu = Hierarchy(ml, enb, roi=roi)
    gpu.set_tma_staging(tma)
    orc = COracle(ml, enb, roi=roi)
    load_random([gpu, orc], ml, enb, seed=7)
    for l in range(ml):
        for impl in (gpu, orc):
            impl.internal_force(l, U, RU, 1e-5)
        assert rel(gpu.get(RU, l), orc.get(RU, l)) < 1e-12, l
    for l in range(ml + 1):
        for impl in (gpu, orc):
            impl.fld(l, D, R, 2.0)
        assert rel(gpu.get(R, l), orc.get(R, l)) < 1e-12, l
        for impl in (gpu, orc):
            impl.fd_h(l)
    for impl in (gpu, orc):
        impl.phase_field((3, 2, 1, 1, 1), 2.0, 1, 1.0, pf_tol=1e-30)
    for f in (D, R, FD):
        assert rel(gpu.get(f, ml), orc.get(f, ml)) < 1e-10, f
    for t in (0, 1):
        for impl in (gpu, orc):
            impl.u_entire((3, 2, 1, 1, 1), 1e-5, 1.0, t, 1.0, mech_tol=1e-30)
        for f in (U, RU, FU):
            assert rel(gpu.get(f, ml), orc.get(f, ml)) < 1e-10, (t, f)
    gpu.close()
    orc.close()
