"""Where the second copies of the run paths are allocated, on the host alone."""
import pytest

torch = pytest.importorskip("torch")


class _Queue:
    """Stands for a stream; what is allocated while it is current is recorded."""

    def __init__(self):
        self.current = False

    def __enter__(self):
        self.current = True

    def __exit__(self, *exc):
        self.current = False


def _simulation():
    from opencl_fdtd_gb300.simulation import Simulation
    sim = Simulation.__new__(Simulation)
    sim._plan = None
    sim._scratch = None
    sim.queue = _Queue()
    sim.E, sim.H = torch.zeros(6), torch.zeros(6)
    sim.psi = {k: [(torch.zeros(2), torch.zeros(2))] for k in "EH"}
    return sim


@pytest.mark.parametrize("modes,count", [(("hs",), 3), (("ahead",), 6), (("hs", "ahead"), 6), (("fused",), 6)])
def test_copies_are_allocated_on_the_queue(monkeypatch, modes, count):
    sim = _simulation()
    on_queue = []
    empty_like = torch.empty_like

    def recorded(t, **kw):
        on_queue.append(sim.queue.current)
        return empty_like(t, **kw)
    monkeypatch.setattr(torch.cuda, "stream", lambda q: q)
    monkeypatch.setattr(torch, "empty_like", recorded)
    for mode in modes:
        sim._ensure_scratch(mode)
    assert on_queue == [True] * count
    assert not sim.queue.current
