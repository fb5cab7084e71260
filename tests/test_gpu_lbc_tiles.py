"""The learned boundary at the edges of its kernels' tiles (2 x 16 columns a warp) and with every
arrangement of learned faces, sources on and off the learned planes: run() (launches that may overlap,
sources inside the E launch where the fix-up leaves their cells alone) against the single calls, bit for
bit; and the tensor-core prediction against float32 on the same weights."""
import math

import numpy
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _net(L, seed):
    net = L.BoundaryNet(seed=seed)
    rng = numpy.random.default_rng(seed)
    net.params += torch.from_numpy((0.02 * rng.standard_normal(tuple(net.params.shape))).astype(numpy.float32)).cuda()
    net._packed = None
    return net


def _kw(shape, seed, poynting):
    rng = numpy.random.default_rng(seed)
    return dict(epsilon=[rng.uniform(1, 4, shape).astype(numpy.float32) for _ in range(3)], pmls=[], do_poynting=poynting,
                initial_fields={k: [0.1 * rng.standard_normal(shape).astype(numpy.float32) for _ in range(3)] for k in "EH"},
                dt=0.99 / math.sqrt(3))


@pytest.mark.parametrize("faces", [["+z"], ["-x"], ["+y", "-z"], ["-x", "+x", "-y", "+y", "-z", "+z"]])
@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 17, 16), (5, 6, 33), (18, 9, 31)])
@pytest.mark.parametrize("poynting", [False, True])
def test_run_equals_single_calls(shape, faces, poynting):
    from opencl_fdtd_gb300 import Simulation, learned_boundary as L
    lb = L.LearnedBoundary(_net(L, 3), "bf16x2", faces=faces)
    a, b = (Simulation(**_kw(shape, 5, poynting)) for _ in range(2))
    lb.attach(a)
    n = 4
    for cell in (a.N // 2 + shape[2] // 2, 0, a.N - 1):      # inside where there is an inside, two corners
        for src in (cell, cell + 2 * a.N):
            vals = [0.3 * math.sin(0.4 * t + src) for t in range(n)]
            a.run(n, point_sources=[(src, vals)], path="hs" if poynting else "auto")
            for t in range(n):
                lb.step(b, point_sources=[(src, vals[t])])
            assert torch.equal(a.E, b.E) and torch.equal(a.H, b.H), src


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 16, 17), (4, 15, 33), (7, 34, 18)])
@pytest.mark.parametrize("precision,tol", [("bf16x2", 2e-4), ("bf16", 3e-2)])
def test_prediction_at_tile_edges(shape, precision, tol):
    """Both on weights rounded to bfloat16: the activations' rounding (2^-16 and 2^-8 a value, over three
    layers) is the only difference."""
    import ctypes
    from opencl_fdtd_gb300 import learned_boundary as L
    net = _net(L, 8)
    net.params.copy_(net.params.to(torch.bfloat16).to(torch.float32))
    net._packed = None
    rng = numpy.random.default_rng(sum(shape))
    n3 = 3 * int(numpy.prod(shape))
    E, H = (torch.from_numpy(rng.standard_normal(n3).astype(numpy.float32)).cuda() for _ in range(2))
    cols, _ = L.columns(shape, 63)
    out = []
    for prec in ("f32", precision):
        pred = torch.zeros((cols, 6), device="cuda")
        L._lib.check(L._lib.load().fdtd_lbc_predict(
            L._shape_arg(shape), 63, -1, L.PRECISIONS[prec], 0.0, net.weights(prec).data_ptr(), E.data_ptr(), H.data_ptr(),
            pred.data_ptr(), pred.numel(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        out.append(pred.double())
    assert (out[0] - out[1]).abs().max() <= tol * out[0].abs().max()
