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
    sim._refused = False
    sim.device = None
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


def test_refused_copies_are_tried_again_when_there_is_room(monkeypatch):
    """36 float32 values are missing: E, H and four CPML arrays."""
    sim = _simulation()
    sim.E, sim.H = torch.zeros(12), torch.zeros(12)
    sim.psi = {k: [(torch.zeros(2), torch.zeros(4))] for k in "EH"}
    tries, state = [], {"free": 0, "reserved": 1000, "allocated": 1000, "fits": False}
    empty_like = torch.empty_like

    def allocate(t, **kw):
        tries.append(t.numel())
        if not state["fits"] and len(tries) % 2 == 0:
            raise torch.cuda.OutOfMemoryError("no room")
        return empty_like(t, **kw)
    monkeypatch.setattr(torch.cuda, "stream", lambda q: q)
    monkeypatch.setattr(torch, "empty_like", allocate)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda d: (state["free"], 10000))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda d: state["reserved"])
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda d: state["allocated"])
    assert not sim._try_scratch("ahead") and len(tries) == 2
    for _ in range(3):
        assert not sim._try_scratch("ahead") and len(tries) == 2
    state["free"] = 36 * 4 - 1
    assert not sim._try_scratch("ahead") and len(tries) == 2
    state.update(reserved=1001, fits=True)
    assert sim._try_scratch("ahead") and len(tries) == 8
    state.update(free=0, reserved=1000)
    assert sim._try_scratch("ahead") and len(tries) == 8
