"""A server that builds its own contexts admits from the start, and builds none but its requests' (CPU)."""
from hpcrack_b200 import serving as sv
from test_serving_host import FakeSolver, _req


def test_default_factory_admits_at_once(monkeypatch):
    made = []
    monkeypatch.setattr(sv, "default_factory", lambda device=0, tma=True: lambda w: made.append(w.name) or FakeSolver(w))
    srv = sv.SolveServer(hbm_budget=100, slots=2)
    res = srv.replay([_req(0, 9, increments=1), _req(1, 9, increments=1)])
    assert sorted(made) == ["r0", "r1"]
    assert max(r.admitted for r in res) < 0.09
    assert FakeSolver.live == 0
