import os
import sys
import time

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); parity tests of the CUDA library")
    config.addinivalue_line("markers", "slow: longer CPU test")


def _has_gpu() -> bool:
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


def pytest_collection_modifyitems(config, items):
    if _has_gpu():
        return
    skip = pytest.mark.skip(reason="no CUDA device on this machine")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)


@pytest.fixture(autouse=True)
def runs_of_a_mix_start_together(request, monkeypatch):
    """test_same_result_alone_and_in_mix compares requests run alone with the same ones run side by side.  They arrive
    50 ms apart and the first takes 21 ms on a B200, so by themselves they would run one after the other: for this test
    the slots open once all three have arrived."""
    if request.node.name != "test_same_result_alone_and_in_mix":
        return
    from hpcrack_b200 import serving
    admit = serving.SolveServer._admit

    def admit_after_the_last_arrival(server):
        time.sleep(max(0.0, 0.11 - server.now()))
        return admit(server)

    monkeypatch.setattr(serving.SolveServer, "_admit", admit_after_the_last_arrival)
