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
    assert a._overlap == overlap
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
        assert b.tuning("last_run_ahead") == 0
        assert b.tuning("last_run_path") == (2 if poynting else 1)
    _same(a, b)
    assert (b._scratch is None) == (not poynting)
    if poynting:
        assert b._scratch[0] is None and b._scratch[1] is not None


def _graded(shape, rng=numpy.random.default_rng(2)):
    return [[rng.uniform(0.8, 1.25, n) for n in shape] for _ in range(2)]


@pytest.mark.parametrize("dx", ["unit", "half", "table"])
@pytest.mark.parametrize("mu", [False, True])
@pytest.mark.parametrize("poynting", [True, False])
def test_ahead_is_the_path_that_runs(dx, mu, poynting):
    """'ahead' and 'hs' share their path code: the launches that make the next step's E are told apart."""
    shape, kw = (14, 11, 300), {}
    if dx != "unit":
        kw["dxes"] = 0.5 if dx == "half" else _graded(shape)
    if mu:
        kw["mu"] = [numpy.full(shape, 1.5, numpy.float32)] * 3
    faces = [(a, p, 3) for a in "xyz" for p in "np"]
    a, b = _sim(shape, faces, poynting, **kw), _sim(shape, faces, poynting, **kw)
    _loop(a, 6)
    b.run(5, path="ahead")
    assert b.tuning("last_run_ahead") == 1 and b.tuning("last_run_path") == 2
    b.run(1, path="ahead")
    assert b.tuning("last_run_ahead") == 0
    _same(a, b)


@pytest.mark.parametrize("shape,poynting,path,ahead", [
    ((24, 24, 24), True, 2, 1), ((24, 24, 24), False, 1, 0), ((64, 64, 64), True, 2, 0), ((64, 64, 64), False, 1, 0),
    ((180, 150, 90), True, 2, 1), ((180, 150, 90), False, 2, 1),
])
def test_automatic_path(shape, poynting, path, ahead):
    """By cells and L2: the lines of Simulation._auto_path for an L2 of about 130 MB."""
    l2 = torch.cuda.get_device_properties(0).L2_cache_size
    if not 115e6 < l2 < 144e6:
        pytest.skip("the lines are those of another L2")
    sim = _sim(shape, [(a, p, 4) for a in "xyz" for p in "np"], poynting)
    sim.run(3)
    assert (sim.tuning("last_run_path"), sim.tuning("last_run_ahead")) == (path, ahead)
    double = _sim((24, 24, 24), (("x", "n", 4),), poynting, float_type=numpy.float64)
    double.run(3)
    assert (double.tuning("last_run_path"), double.tuning("last_run_ahead")) == (1, 0)


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 1, 2), (3, 1, 1), (1, 5, 37), (2, 3, 511), (1, 1, 4096), (2, 1, 10007)])
@pytest.mark.parametrize("mu", [False, True])
def test_rows_of_any_length(shape, mu):
    """Tiles of whole and of divided rows, down to one cell."""
    kw = {"mu": [numpy.full(shape, 1.5, numpy.float32)] * 3} if mu else {}
    faces = [("z", p, 8) for p in "np"] if shape[2] > 100 else []
    a, b = _sim(shape, faces, **kw), _sim(shape, faces, **kw)
    _loop(a, 5)
    b.run(5, path="ahead")
    assert b.tuning("last_run_ahead") == 1
    _same(a, b)


def test_a_long_row_costs_the_host_no_time():
    """20 million cells in a row: finding the tiles takes microseconds, not a try of every division."""
    import time
    one = numpy.ones((1, 1, 20_000_000), numpy.float32)
    from opencl_fdtd_gb300 import Simulation
    sim = Simulation([one] * 3, [], do_poynting=False)
    sim.run(2, path="ahead")
    took = []
    for _ in range(10):
        torch.cuda.synchronize()
        t = time.perf_counter()
        sim.run(2, path="ahead")
        took.append(time.perf_counter() - t)
    assert sim.tuning("last_run_ahead") == 1
    assert min(took) < 1e-3
