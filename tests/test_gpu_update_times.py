"""Single updates against each other on one grid, where a form of a kernel once cost more than what it
adds: times of the same launches on the same GPU, the shortest of several."""
import numpy
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

SHAPE = (200, 200, 200)


def _sim(dtype=numpy.float32, mu=False, shape=SHAPE, faces="xyz", **kw):
    from opencl_fdtd_gb300 import Simulation
    one = numpy.ones(shape, dtype)
    if mu:
        kw["mu"] = [one] * 3
    return Simulation([one] * 3, [{"axis": a, "polarity": p, "thickness": 8} for a in faces for p in "np"],
                      do_poynting=False, float_type=dtype, **kw)


def _time(update):
    best = float("inf")
    for _ in range(8):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        update([])
        torch.cuda.synchronize()
        torch.cuda._sleep(400_000)                           # the launches are queued before the first runs
        a.record()
        for _ in range(6):
            update([])
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) / 6)
    return best


def test_h_with_mu():
    """Reading dt/mu makes 12 arrays of 9 in H, a third more bytes at most; the kernel is far from the
    memory's limit and takes 1.09 times as long. Loading each plane only when it is updated took 1.27."""
    assert _time(_sim(mu=True).update_H) <= 1.18 * _time(_sim().update_H)


def test_h_beside_e_in_double():
    """H without the products does what E does, on 9 arrays instead of 12: as long as E at most, with room for
    the scatter of the times. One plane a thread took 1.27 times as long."""
    sim = _sim(numpy.float64)
    assert _time(sim.update_H) <= 1.18 * _time(sim.update_E)


def test_e_of_bloch_pairs_on_graded_cells():
    """The spacings more to read: 1.03 times E on unit cells. With the cells outside the z faces
    first, on rows that are not whole sectors, it took 1.15 times as long."""
    shape = (33, 700, 300)
    kw = dict(shape=shape, faces="z", bloch_boundaries=[{"axis": "x", "real": 0.6, "imag": 0.8}])
    graded = [[numpy.ones(n) for n in shape] for _ in range(2)]
    assert _time(_sim(dxes=graded, **kw).update_E) <= 1.09 * _time(_sim(**kw).update_E)
