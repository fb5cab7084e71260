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
