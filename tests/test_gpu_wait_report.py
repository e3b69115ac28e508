"""Every entry point that launches kernels with bounded waits reports a wait that ran out (GPU).

Such a kernel stops, sets the context's flag and leaves the rest of its output unwritten.  The flag is set here from
the host, as a kernel sets it; the call that finds it returns an error and clears it, so that the
next call is not blamed.
"""
import ctypes as C

import pytest

from hpcrack_b200 import lib as L
from hpcrack_b200.solver import Hierarchy, RU, U
from cases import D, R, load_random

pytestmark = pytest.mark.gpu
MG = (4, 1, 1, 1, 1)

CALLS = {
    "internal_force_coarse": lambda h: h.internal_force(0, U, RU, 1e-5),
    "internal_force_finest": lambda h: h.internal_force(1, U, RU, 1e-5),
    "fld": lambda h: h.fld(1, D, R, 2.0),
    "initial_residual_u": lambda h: h.initial_residual_u(0, 1e-5),
    "initial_residual_d": lambda h: h.initial_residual_d(1, 2.0),
    "pcg_u": lambda h: h.pcg_u(0, 1e-5, 1.0, 2, 1, 1.0),
    "pcg_d": lambda h: h.pcg_d(1, 2.0, 2, 1, 1.0),
    "cycle_u": lambda h: h.cycle_u(1, MG, 1e-5, 1.0, 1, 1.0),
    "cycle_d": lambda h: h.cycle_d(1, MG, 2.0, 1, 1.0),
    "u_entire": lambda h: h.u_entire(MG, 1e-5, 1.0, 1, 1.0, mech_tol=1e-30),
    "phase_field": lambda h: h.phase_field(MG, 2.0, 1, 1.0, pf_tol=1e-30),
}


@pytest.mark.parametrize("name", CALLS)
def test_call_reports_and_clears(name):
    set_wait_error = L.load()._ZN3hpc14set_wait_errorEP7hpc_ctx  # hpc::set_wait_error(hpc_ctx*)
    set_wait_error.argtypes, set_wait_error.restype = [C.c_void_p], None
    enb = (4, 3, 5)
    with Hierarchy(1, enb) as h:
        load_random([h], 1, enb, seed=2)
        set_wait_error(h.h)
        with pytest.raises(Exception, match="bounded wait"):
            CALLS[name](h)
        CALLS[name](h)
