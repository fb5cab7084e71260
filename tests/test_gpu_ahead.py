"""run(path='ahead'): one launch per step that makes H and S of the step and E of the next. The tiles'
edges (row segments, halo rows and columns, z-face columns on threads of their own), the chunk's first
evaluated plane, the swaps of the copies and the forms (spacing, mu, Poynting off) against the
per-update kernels, bit for bit: both evaluate the same expressions in the same order."""
import copy
import math

import numpy
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _kwargs(shape, faces, seed, **extra):
    rng = numpy.random.default_rng(seed)
    eps = [rng.uniform(1, 4, shape).astype(numpy.float32) for _ in range(3)]
    eps[1][shape[0] // 2, shape[1] // 2, shape[2] // 2] = numpy.inf
    kw = dict(epsilon=eps, pmls=[{"axis": f[0], "polarity": f[1], "thickness": t} for f, t in faces],
              initial_fields={k: [rng.standard_normal(shape).astype(numpy.float32) for _ in range(3)] for k in "EH"},
              do_poynting=True)
    kw.update(extra)
    return kw


def _pair(kw, nsteps, sources, tune=None, monitor=False):
    from opencl_fdtd_gb300 import Simulation
    sims, mons = [], []
    for path in ("plain", "ahead"):
        s = Simulation(**copy.deepcopy(kw))
        if tune and path == "ahead":
            s.tune(**tune)
        m = s.dft_monitor([1, s.N + 2], [0.3, 0.4]) if monitor else None
        for n in nsteps:
            s.run(n, point_sources=[(i, v[:n]) for i, v in sources(s.N)], path=path, monitor=m)
        sims.append(s)
        mons.append(m)
    a, b = sims
    assert b.tuning("last_run_path") == 2
    for k in ("E", "H", "S", "oS"):
        if getattr(a, k) is not None:
            assert torch.equal(getattr(a, k), getattr(b, k)), k
    for k in "EH":
        for (u, v), (p, q) in zip(a.psi[k], b.psi[k]):
            assert torch.equal(u, p) and torch.equal(v, q), ("psi", k)
    if monitor:
        assert numpy.array_equal(mons[0].series(), mons[1].series())
        assert torch.equal(mons[0].accum, mons[1].accum)


def _one_source(N):
    return [(N + N // 2, [math.sin(0.4 * t) for t in range(8)])]


ALL6 = ("xn", "xp", "yn", "yp", "zn", "zp")


def _six(t):
    return [(f, t) for f in ALL6]


# z extents around the segment lengths (37 cells and more), one cell, whole rows in the faces
@pytest.mark.parametrize("shape,faces", [
    ((5, 4, 1), []), ((1, 1, 1), []), ((1, 5, 40), [("zn", 3)]), ((3, 2, 36), _six(1)), ((6, 5, 37), [("zp", 4)]),
    ((6, 7, 73), _six(2)), ((4, 30, 74), [("zn", 37), ("zp", 37)]), ((5, 9, 75), [("zn", 38), ("zp", 1)]),
    ((4, 13, 111), [("zn", 40), ("zp", 5), ("yp", 13)]), ((7, 6, 223), _six(3)), ((5, 26, 224), [("zn", 112)]),
    ((6, 5, 300), _six(2)), ((5, 4, 511), [("zp", 511)]), ((17, 50, 20), [("yn", 6), ("xp", 5)]),
    ((26, 14, 38), [("zn", 1), ("zp", 37), ("xn", 26)])])
@pytest.mark.parametrize("nsteps", [(1,), (2,), (3, 4)])
def test_ahead_tiles_equal_per_update_kernels(shape, faces, nsteps):
    _pair(_kwargs(shape, faces, sum(shape) + len(faces)), nsteps, _one_source)


@pytest.mark.parametrize("tune", [dict(hs_xchunk=1), dict(hs_xchunk=2), dict(hs_xchunk=5, pdl=False), dict(hs_xchunk=64),
                                  dict(hs_reverse=False, hs_dft=False)])
def test_ahead_launch_options_and_monitor(tune):
    _pair(_kwargs((13, 12, 41), _six(3), 3), (4, 3), _one_source, tune=tune, monitor=True)


def _extra(form, shape):
    rng = numpy.random.default_rng(5)
    return {"half": dict(dxes=0.5), "tables": dict(dxes=[[rng.uniform(0.8, 1.25, n) for n in shape] for _ in range(2)]),
            "mu": dict(mu=[rng.uniform(1, 2, shape).astype(numpy.float32) for _ in range(3)]), "unit": {}}[form]


@pytest.mark.parametrize("poynting", [True, False])
@pytest.mark.parametrize("form", ["unit", "half", "tables", "mu"])
def test_ahead_forms(form, poynting):
    shape = (11, 15, 39)
    kw = _kwargs(shape, _six(4), 9, do_poynting=poynting, **_extra(form, shape))
    _pair(kw, (1, 2, 5), _one_source)


@pytest.mark.parametrize("count", [3, 11])
def test_ahead_point_sources(count):
    """Up to 8 sources inside the launch, in list order (two on one cell), more after it."""
    def sources(N):
        rng = numpy.random.default_rng(count)
        cells = [int(i) for i in rng.integers(0, 3 * N, count - 1)]
        return [(i, [float(v) for v in rng.standard_normal(6)]) for i in cells + cells[:1]]
    _pair(_kwargs((9, 10, 38), _six(2), 4), (6, 5), sources)


def test_auto_path_choice():
    """Poynting on: 'ahead' from two steps on, but 'hs' where launches no longer count and the fields fit
    the L2; off: per-update kernels while they fit; double precision and Bloch boundaries: per-update."""
    from opencl_fdtd_gb300 import Simulation
    kw = _kwargs((8, 8, 8), _six(2), 1)
    s = Simulation(**copy.deepcopy(kw))
    assert (s._auto_path(1), s._auto_path(2)) == ("hs", "ahead")
    mid = Simulation(**_kwargs((60, 50, 40), _six(2), 1))
    assert mid._auto_path(2) == "hs"
    mid.run(3)
    assert mid.tuning("last_run_path") == 2
    kw["do_poynting"] = False
    assert Simulation(**copy.deepcopy(kw))._auto_path(5) == "plain"
    kw["float_type"] = numpy.float64
    kw["do_poynting"] = True
    d = Simulation(**kw)
    assert d._auto_path(5) == "plain"
    d.run(2, path="ahead")                       # no such form in double precision: H and S in one launch
    assert d.tuning("last_run_path") == 2
