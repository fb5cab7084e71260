"""Batches through the C ABI, with variants that a Simulation does not make."""
import ctypes

import numpy
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


class _Batch:
    """Float32 variants of these shapes, unit cells, no faces; one source, one monitor point each."""

    def __init__(self, shapes, rows):
        from opencl_fdtd_gb300 import _lib
        self.lib, self.check = _lib.load(), _lib.check
        self.handle = ctypes.c_void_p()
        arr = (_lib.FdtdBatchVariant * len(shapes))()
        self.fields, self.series, self.keep = [], [], []
        for d, shape in zip(arr, shapes):
            n = 3 * shape[0] * shape[1] * shape[2]
            gen = torch.Generator(device="cuda").manual_seed(n)
            E, H, ce = (torch.randn(n, generator=gen, device="cuda") for _ in range(3))
            ce.abs_().mul_(0.1)
            values = torch.arange(rows, device="cuda", dtype=torch.float32) + 1
            ser = torch.zeros((rows, 1), dtype=torch.float64, device="cuda")
            d.shape[:] = shape
            d.dt, d.dx = 0.5, 1.0
            d.E, d.H, d.ce = E.data_ptr(), H.data_ptr(), ce.data_ptr()
            d.n_src = d.n_mon = 1
            d.src_index[0] = d.mon_index[0] = n // 2
            d.src_values, d.series = values.data_ptr(), ser.data_ptr()
            self.fields.append((E, H))
            self.series.append(ser)
            self.keep += [ce, values]
        torch.cuda.synchronize()
        self.check(self.lib.fdtd_batch_create(arr, len(shapes), _lib.FDTD_STORE_F32, rows, ctypes.byref(self.handle)))

    def run(self, n, stream=None):
        st = stream.cuda_stream if stream is not None else torch.cuda.current_stream().cuda_stream
        self.check(self.lib.fdtd_batch_run(self.handle, ctypes.c_void_p(st), n))

    def state(self):
        torch.cuda.synchronize()
        return [t.clone() for pair in self.fields for t in pair] + [s.clone() for s in self.series]

    def close(self):
        torch.cuda.synchronize()
        self.lib.fdtd_batch_destroy(self.handle)


def _result(shapes, steps, persistent=False, xchunk=None):
    from opencl_fdtd_gb300 import _lib
    b = _Batch(shapes, sum(steps))
    if persistent:
        b.check(b.lib.fdtd_batch_schedule(b.handle, _lib.FDTD_BATCH_PERSISTENT))
    if xchunk is not None:
        b.check(b.lib.fdtd_batch_tune(b.handle, xchunk, 0))
    for n in steps:
        b.run(n)
    out = b.state()
    b.close()
    return out


@pytest.mark.parametrize("shape,xchunk", [((70000, 4, 2), 1), ((600000, 1, 1), None), ((65535, 4, 2), 1)])
def test_more_planes_than_a_grid_has_rows(shape, xchunk):
    """A variant launched alone puts its chunks of planes on the grid's y extent, which ends at 65535; the
    persistent schedule has no such limit."""
    for a, b in zip(_result([shape], (2, 1), xchunk=xchunk), _result([shape], (2, 1), persistent=True)):
        assert torch.equal(a, b)


def test_automatic_tiles_can_be_asked_for_again():
    """A tile length of 0 is the automatic one: the same launches, and the same tile list, which a
    captured run refers to, as before the batch was tuned to what it had chosen."""
    shapes, steps = [(128, 72, 64), (64, 64, 37), (80, 80, 80)], (1, 2)
    ref = _result(shapes, steps)
    for chunks in ((0,), (3, 0), (8, 0)):
        b = _Batch(shapes, sum(steps))
        for c in chunks:
            b.check(b.lib.fdtd_batch_tune(b.handle, c, 0))
        for n in steps:
            b.run(n)
        out = b.state()
        b.close()
        for x, y in zip(ref, out):
            assert torch.equal(x, y)
    # 25 blocks a plane and 238 planes that share launches, far more than the GPU holds: 8 planes a tile
    shapes = [(80, 79, 79), (79, 80, 79), (79, 79, 80)]
    ref = _result(shapes, steps)
    b = _Batch(shapes, sum(steps))
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        b.run(1, stream)
    b.check(b.lib.fdtd_batch_tune(b.handle, 8, 0))
    b.check(b.lib.fdtd_batch_tune(b.handle, 0, 0))
    for _ in range(sum(steps)):
        graph.replay()
    for x, y in zip(ref, b.state()):
        assert torch.equal(x, y)
    del graph
    b.close()


def _simulations():
    from opencl_fdtd_gb300 import Simulation
    sims = []
    for shape in ((84, 77, 79), (12, 10, 9)):
        rng = numpy.random.default_rng(shape[0])
        sims.append(Simulation([rng.uniform(1, 4, shape).astype(numpy.float32) for _ in range(3)], [], do_poynting=False,
                               initial_fields={k: [rng.standard_normal(shape).astype(numpy.float32) for _ in range(3)]
                                               for k in "EH"}))
    return sims


def test_tune_keeps_the_automatic_tiles():
    from opencl_fdtd_gb300.batch import BatchSimulation
    b = BatchSimulation(_simulations())
    assert b.xchunk == 0
    b.tune(schedule="persistent")
    b.tune(schedule="launches")
    assert b.xchunk == 0
    b.tune(xchunk=5)
    b.tune(blocks_per_sm=1)
    assert b.xchunk == 5
    b.tune(xchunk=0)
    assert b.xchunk == 0


def test_autotune_times_the_automatic_tiles(monkeypatch):
    from opencl_fdtd_gb300 import autotune
    from opencl_fdtd_gb300.batch import BatchSimulation
    b = BatchSimulation(_simulations())
    monkeypatch.setattr(autotune, "_MEMO", {})
    monkeypatch.setattr(autotune, "time_config",
                        lambda batch, xc, blocks, steps, sched: 1.0 if (xc, sched) == (0, "launches") else 2.0)
    choice = b.autotune(steps=1)
    assert (choice["xchunk"], choice["schedule"]) == (0, "launches") and b.xchunk == 0
    assert b.autotune(steps=1)["cached"] and b.xchunk == 0


def test_captured_run_with_a_variant_launched_alone():
    """The descriptor of such a variant is in the captured launches themselves."""
    from opencl_fdtd_gb300.batch import BatchSimulation
    ref, sims = _simulations(), _simulations()
    BatchSimulation(ref).run(6)
    b = BatchSimulation(sims)
    b.capture(2)
    for _ in range(3):
        b.replay()
    torch.cuda.synchronize()
    assert b.step_counter() == 6
    for x, y in zip(ref, sims):
        assert torch.equal(x.E, y.E) and torch.equal(x.H, y.H)
    assert b.step_launches() == 4
    b.tune(schedule="persistent")
    assert b.step_launches() == 0


@pytest.mark.parametrize("shapes,length,launches", [
    ([(48, 47, 45)], 1, 2),                                  # 432 blocks for the GPU's 608 places
    ([(48, 47, 45), (165, 150, 73)], 1, 4),                  # beside a variant launched alone: the same
    ([(48, 47, 45)] * 4, 2, 2),
    ([(80, 79, 79), (79, 80, 79), (79, 79, 80)], 8, 2),
])
def test_shared_launches_hold_their_own_variants(shapes, length, launches):
    from opencl_fdtd_gb300 import _lib
    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("the lengths are those of 152 SMs")
    b = _Batch(shapes, 1)
    v = ctypes.c_int32()
    for key, want in ((_lib.FDTD_BATCH_GET_XCHUNK, 0), (_lib.FDTD_BATCH_GET_TILE_XCHUNK, length),
                      (_lib.FDTD_BATCH_GET_STEP_LAUNCHES, launches)):
        b.check(b.lib.fdtd_batch_get(b.handle, key, ctypes.byref(v)))
        assert v.value == want, key
    b.close()
