"""Batched stepping with the tile length it chooses itself (small batches: down to one plane), with
sources and monitors on the tiles' first and last cells and planes, x faces that end inside a tile and
cells that are not unit cells: the same bits as each variant on its own; 16-bit storage without
exponents equal to the variant stepped alone in the same storage."""
import copy
import math

import numpy
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

# (shape, thickness of the x, y, z faces); 256 cells and 8 planes are a full tile
VARIANTS = [((24, 16, 16), (3, 2, 4)), ((8, 8, 32), (4, 4, 0)), ((7, 85, 3), (1, 5, 1)), ((17, 51, 5), (0, 9, 2)),
            ((9, 1, 257), (2, 0, 60)), ((1, 20, 20), (0, 3, 3))]


def _kw(shape, T, seed, dx):
    rng = numpy.random.default_rng(seed)
    return dict(epsilon=[rng.uniform(1, 6, shape).astype(numpy.float32) for _ in range(3)],
                pmls=[{"axis": a, "polarity": p, "thickness": t} for a, t in zip("xyz", T) for p in "np" if t],
                initial_fields={k: [0.1 * rng.standard_normal(shape).astype(numpy.float32) for _ in range(3)] for k in "EH"},
                do_poynting=False, **({"dxes": dx} if dx != 1.0 else {}))


def _points(shape):
    """Flat indices on the edges of tiles: first and last cell and plane, cells 255 and 256 of a plane."""
    nx, syz = shape[0], shape[1] * shape[2]
    N = nx * syz
    cells = {0, N - 1, min(255, syz - 1), min(256, syz - 1) + (min(8, nx) - 1) * syz, min(8, nx - 1) * syz}
    return sorted(c + comp * N for comp, c in enumerate(sorted(cells)[:3])) + [sorted(cells)[-2]]


@pytest.mark.parametrize("storage", ["f32", "bf16u", "bf16"])
@pytest.mark.parametrize("dx", [1.0, 0.5])
@pytest.mark.parametrize("schedule", ["launches", "persistent"])
def test_tiles_equal_single_variants(storage, dx, schedule):
    from opencl_fdtd_gb300 import Simulation, _lib
    from opencl_fdtd_gb300.batch import BatchSimulation
    kws = [_kw(s, t, i, dx) for i, (s, t) in enumerate(VARIANTS)]
    n = 5

    def step(group):
        sims = [Simulation(**copy.deepcopy(kws[i])) for i in group]
        pts = [_points(VARIANTS[i][0]) for i in group]
        src = [[(p, [math.sin(0.3 * t + k) for t in range(n)]) for k, p in enumerate(ps)] for ps in pts]
        b = BatchSimulation(sims, storage=storage, sources=src, monitors=pts, steps=n)
        _lib.check(b._lib.fdtd_batch_schedule(b._batch, _lib.FDTD_BATCH_LAUNCHES if schedule == "launches"
                                              else _lib.FDTD_BATCH_PERSISTENT))
        b.run(n)
        b.sync()
        return sims, [t.cpu().numpy() for t in b.series]
    together, series = step(range(len(kws)))
    for i in range(len(kws)):
        (alone,), (one,) = step([i])
        if storage == "f32":
            ref = Simulation(**copy.deepcopy(kws[i]))
            ref.run(n, point_sources=[(p, [math.sin(0.3 * t + k) for t in range(n)])
                                      for k, p in enumerate(_points(VARIANTS[i][0]))], path="plain")
            assert torch.equal(ref.E, alone.E) and torch.equal(ref.H, alone.H)
        assert torch.equal(together[i].E, alone.E) and torch.equal(together[i].H, alone.H)
        assert numpy.array_equal(series[i], one)


@pytest.mark.parametrize("dx,chunk", [(1.0, None), (0.5, 3), (1.0, 64)])
def test_large_variants_launched_alone(dx, chunk):
    """From half a million cells on a float32 variant has launches of its own; beside smaller ones, which
    share theirs."""
    from opencl_fdtd_gb300 import Simulation
    from opencl_fdtd_gb300.batch import BatchSimulation
    cases = [((12, 10, 9), (2, 0, 3)), ((84, 77, 79), (5, 4, 8)), ((7, 85, 3), (1, 5, 1)), ((65, 64, 125), (0, 8, 1))]
    kws = [_kw(s, t, 20 + i, dx) for i, (s, t) in enumerate(cases)]
    pts = [_points(s) for s, _ in cases]
    n = 5
    src = [[(p, [math.sin(0.3 * t + k) for t in range(n)]) for k, p in enumerate(ps)] for ps in pts]
    sims = [Simulation(**copy.deepcopy(kw)) for kw in kws]
    b = BatchSimulation(sims, storage="f32", sources=src, monitors=pts, steps=n)
    if chunk:
        b.tune(xchunk=chunk)
    b.run(2)
    b.run(3)
    torch.cuda.synchronize()
    assert b.step_counter() == n
    for kw, sim, ps, ss, ser in zip(kws, sims, pts, src, b.series):
        ref = Simulation(**copy.deepcopy(kw))
        m = ref.dft_monitor([(i // ref.N, numpy.unravel_index(i % ref.N, ref.shape)) for i in ps], ())
        ref.run(n, point_sources=ss, monitor=m, path="plain")
        assert torch.equal(ref.E, sim.E) and torch.equal(ref.H, sim.H)
        for f in "EH":
            for (u, v), (p, q) in zip(ref.psi[f], sim.psi[f]):
                assert torch.equal(u, p) and torch.equal(v, q)
        assert numpy.array_equal(m.series(), ser.cpu().numpy())
