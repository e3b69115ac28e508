"""Where no cluster of the small-level smoother's size can be resident, the per-iteration kernels run (GPU).

A device may offer fewer SMs side by side than the cluster has blocks (a partitioned GPU).  The occupancy query is
answered "none" by a library put in front of the CUDA runtime, in a process of its own; the solve there must
equal, bit for bit and launch for launch, one with the cluster smoother switched off.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))

NONE = """
int cudaOccupancyMaxActiveClusters(int* n, const void* f, const void* cfg) { (void)f; (void)cfg; *n = 0; return 0; }
"""
SOLVE = """
import hashlib, sys
sys.path[:0] = [{root!r}, {here!r}]
from hpcrack_b200.solver import Hierarchy, U
from cases import D, load_random
h = Hierarchy(1, (8, 8, 8))
h.set_fused_coarsest({fused})
load_random([h], 1, (8, 8, 8), seed=3)
n0 = h.launch_count()
h.u_entire((6, 2, 2, 1, 1), 1e-5, 0.5, 1, 1.0, mech_tol=1e-30)
h.phase_field((6, 2, 2, 1, 1), 2.0, 1, 1.0, pf_tol=1e-30)
h.u_entire_fcg((6, 2, 2, 1, 1), 1e-5, 0.5, 1, 1.0, mech_tol=1e-30, mixed=True)
print(h.launch_count() - n0, hashlib.sha256(h.get(U, 1).tobytes() + h.get(D, 1).tobytes()).hexdigest())
"""


def _run(fused, preload=None):
    env = dict(os.environ)
    if preload:
        env["LD_PRELOAD"] = str(preload)
    code = SOLVE.format(root=os.path.dirname(HERE), here=HERE, fused=fused)
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, env=env, timeout=300)
    assert out.returncode == 0, out.stderr
    return out.stdout.split()


def test_no_resident_cluster(tmp_path):
    src, so = tmp_path / "none.c", tmp_path / "none.so"
    src.write_text(NONE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src)], check=True)
    off = _run(False)
    assert _run(True, preload=so) == off
    assert _run(True)[0] != off[0]  # the query matters: with clusters there are fewer launches
