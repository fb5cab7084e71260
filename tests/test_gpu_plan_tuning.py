"""Tuning keys of a plan: read, changed and restored, a key is what it was."""
import numpy
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _sim(dtype):
    from opencl_fdtd_gb300 import Simulation
    rng = numpy.random.default_rng(3)
    shape = (21, 18, 35)
    return Simulation([rng.uniform(1, 4, shape).astype(dtype) for _ in range(3)],
                      [{"axis": "z", "polarity": "n", "thickness": 5}], float_type=dtype,
                      initial_fields={k: [rng.standard_normal(shape).astype(dtype) for _ in range(3)] for k in "EH"})


@pytest.mark.parametrize("dtype", [numpy.float32, numpy.float64])
def test_automatic_planes_per_thread(dtype):
    from opencl_fdtd_gb300 import _lib
    a, b = _sim(dtype), _sim(dtype)
    automatic = a.tuning("xchunk")
    assert automatic == 0
    a.run(3, path="plain")
    a.tune(xchunk=automatic)
    assert a.tuning("xchunk") == automatic
    a.run(2, path="plain")
    b.tune(xchunk=7)
    assert b.tuning("xchunk") == 7
    b.run(5, path="plain")
    assert torch.equal(a.E, b.E) and torch.equal(a.H, b.H) and torch.equal(a.S, b.S)
    for bad in (-1, 4097):
        with pytest.raises(_lib.FdtdError):
            a.tune(xchunk=bad)
