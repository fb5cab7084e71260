"""Which path run() takes, and what it allocates for it."""
import numpy
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _sim(shape=(30, 26, 40), faces=(), poynting=True, **kw):
    from opencl_fdtd_gb300 import Simulation
    rng = numpy.random.default_rng(11)
    return Simulation([rng.uniform(1, 4, shape).astype(numpy.float32) for _ in range(3)],
                      [{"axis": a, "polarity": p, "thickness": t} for a, p, t in faces], do_poynting=poynting,
                      initial_fields={k: [rng.standard_normal(shape).astype(numpy.float32) for _ in range(3)]
                                      for k in "EH"}, **kw)


def _loop(sim, n):
    for _ in range(n):
        sim.update_E([])
        sim.update_H([])
        if sim.update_S:
            sim.update_S([])


def _same(a, b):
    torch.cuda.synchronize()
    for k in "EHS":
        if getattr(a, k) is not None:
            assert torch.equal(getattr(a, k), getattr(b, k)), k


@pytest.mark.parametrize("poynting", [True, False])
@pytest.mark.parametrize("path", ["auto", "ahead"])
@pytest.mark.parametrize("faces,overlap", [
    ((("x", "n", 9), ("x", "p", 8)), True),
    ((("x", "n", 8), ("x", "p", 8)), False),
    ((("x", "n", 9), ("x", "p", 17)), False),                # thicker than its axis: never applies
    ((("y", "p", 4), ("x", "n", 17)), True),
])
def test_overlapping_faces_need_no_copies(faces, overlap, path, poynting):
    shape = (16, 20, 24)
    a, b = _sim(shape, faces, poynting), _sim(shape, faces, poynting)
    assert a._faces_overlap() == overlap
    _loop(a, 4)
    b.run(4, path=path)
    _same(a, b)
    if overlap:
        assert b._scratch is None and b.tuning("last_run_path") == 1


@pytest.mark.parametrize("poynting", [True, False])
def test_no_room_for_the_copies(poynting, monkeypatch):
    """A refused copy of E sends 'ahead' to the path that needs none, with the same results."""
    from opencl_fdtd_gb300 import Simulation
    a, b = _sim(poynting=poynting), _sim(poynting=poynting)
    ensure = Simulation._ensure_scratch

    def refuse(self, mode):
        if mode == "ahead":
            raise torch.cuda.OutOfMemoryError("no room")
        ensure(self, mode)
    monkeypatch.setattr(Simulation, "_ensure_scratch", refuse)
    _loop(a, 7)
    for n in (4, 3):
        b.run(n, path="ahead")
        assert b.tuning("last_run_path") == (2 if poynting else 1)
    _same(a, b)
    assert (b._scratch is None) == (not poynting)
    if poynting:
        assert b._scratch[0] is None and b._scratch[1] is not None
