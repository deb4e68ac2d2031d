"""A unit at the head of the server's queue that waits for room is estimated
once, however often the loop comes by: with FP64 wall layers an estimate is a
pass over the mesh, on the thread that feeds the GPU."""
import hydraphase.serve as serve
from test_serve_logic import FakeHandle, _stream, fake_engine  # noqa: F401


def test_a_waiting_unit_is_estimated_once(fake_engine, monkeypatch):  # noqa: F811
    calls = []

    def estimate(mesh, p):
        calls.append(mesh)
        return 1000 * mesh.neles

    monkeypatch.setattr(serve, "estimate_bytes", estimate)
    reqs = _stream([2, 3, 2, 3], steps=200)
    budget = 1000 * max(r.spec.mesh.neles for r in reqs)
    rep = serve.Server(budget, max_active=4, chunk=5, keep_state=False).run(reqs, realtime=False)
    assert len(rep.results) == 4 and all(r.error is None for r in rep.results) and FakeHandle.peak_live == 1
    assert len(calls) == 4
