"""The boundary network's training kernels at the edges of their tiles (32 samples a block, 256 rows and
16 input rows x 64 or 8 columns a block of the weight gradients), against float64. Tolerances are
forward error bounds: a float32 chain of n terms is off by at most n u times the sum of the terms'
magnitudes (u = 2^-24), and a term carries the roundings of the chains that made it."""
import ctypes

import numpy
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

U = 2.0 ** -24
SIZES = [1, 31, 32, 33, 127, 255, 256, 257, 513]


def _cuda(a):
    return torch.from_numpy(a).cuda()


@pytest.mark.parametrize("B", SIZES)
@pytest.mark.parametrize("weighted", [True, False])
def test_gradient_at_tile_edges(B, weighted):
    from opencl_fdtd_gb300 import _lib, learned_boundary as lb
    rng = numpy.random.default_rng(B)
    net, face = lb.BoundaryNet(seed=B), 3
    flat = _cuda(rng.standard_normal(B * 108 + 1).astype(numpy.float32))
    X = flat[1:].view(B, 108)                    # rows that start off a 16-byte boundary
    T = _cuda(rng.standard_normal((B, 6)).astype(numpy.float32))
    loss, grad = net.gradient(face, X, T, weighted)
    P = net.params[face].double()
    cut = numpy.cumsum([0, 108 * 64, 64, 64 * 64, 64, 64 * 6, 6])
    w1, b1, w2, b2, w3, b3 = (P[cut[i]:cut[i + 1]] for i in range(6))
    w1, w2, w3 = w1.view(108, 64), w2.view(64, 64), w3.view(64, 6)
    gelu = torch.nn.functional.gelu

    def dgelu(a):
        return 0.5 * (1 + torch.erf(a / 2 ** 0.5)) + a * torch.exp(-a * a / 2) / (2 * numpy.pi) ** 0.5
    x, t = X.double(), T.double()
    a1 = x @ w1 + b1
    a2 = gelu(a1) @ w2 + b2
    y = gelu(a2) @ w3 + b3
    wo = net.output_weights(face).double() if weighted else torch.ones(6, dtype=torch.float64, device="cuda")
    dy = 2 * wo * (y - t) / (6 * B)
    d2 = (dy @ w3.T) * dgelu(a2)
    d1 = (d2 @ w2.T) * dgelu(a1)
    ref = torch.cat([v.reshape(-1) for v in (x.T @ d1, d1.sum(0), gelu(a1).T @ d2, d2.sum(0), gelu(a2).T @ dy, dy.sum(0))])
    # magnitudes: the same chain with every sum of absolute values; |gelu(a)| <= |a|, |gelu'| <= 1.13,
    # |gelu''| <= 0.8, so an error of a1 or a2 changes a gradient term by at most that share of it
    m1 = x.abs() @ w1.abs() + b1.abs()
    m2 = m1 @ w2.abs() + b2.abs()
    my = m2 @ w3.abs() + b3.abs()
    n = 108 + 64 + 64 + 6 + 40                   # roundings of the longest chain, erf and exp of a few ulp
    assert ((net.forward(face, X).double() - y).abs() <= 1.13 ** 2 * n * U * my).all()
    md = 2 * wo * (my + t.abs()) / (6 * B)
    k2 = (md @ w3.abs().T) * (1.13 + 0.8 * m2)
    k1 = (k2 @ w2.abs().T) * (1.13 + 0.8 * m1)
    mag = torch.cat([v.reshape(-1) for v in (x.abs().T @ k1, k1.sum(0), m1.T @ k2, k2.sum(0), m2.T @ md, md.sum(0))])
    chain = min(B, 256) + (B + 255) // 256
    assert ((grad.double() - ref).abs() <= (4 * n + chain) * U * mag).all()
    assert abs(float(loss) - float((wo * (y - t) ** 2).mean())) <= (4 * n + 64) * U * float((wo * (my + t.abs()) ** 2).mean())
    again = net.gradient(face, X.clone(), T, weighted)[1].clone()
    assert torch.equal(net.gradient(face, X, T, weighted)[1], again)
    # the same from the two separate calls
    n = ctypes.c_int64()
    _lib.check(_lib.load().fdtd_mlp_backward_workspace(B, ctypes.byref(n)))
    ws, out = (torch.empty(k, dtype=torch.float32, device="cuda") for k in (n.value, lb.NPARAM))
    b = net._buffers(B)
    w = net.output_weights(face).data_ptr() if weighted else None
    _lib.check(_lib.load().fdtd_mlp_backward(net.params[face].data_ptr(), X.data_ptr(), net.forward(face, X).data_ptr(),
                                             T.data_ptr(), w, B, *(b[k].data_ptr() for k in ("A1", "A2", "H1", "H2")),
                                             out.data_ptr(), ws.data_ptr(), ws.numel(), net._stream()))
    assert torch.equal(out, again)


@pytest.mark.parametrize("K,N", [(1, 1), (15, 8), (16, 9), (17, 64), (31, 65), (6, 130), (108, 6), (108, 64)])
@pytest.mark.parametrize("rows", [1, 63, 65, 255, 256, 257, 1030])
def test_gram_at_tile_edges(rows, K, N):
    from opencl_fdtd_gb300 import learned_boundary as lb
    rng = numpy.random.default_rng(rows + K + N)
    A, B = (rng.standard_normal((rows, n)).astype(numpy.float32) for n in (K, N))
    got = lb.BoundaryNet(seed=0).gram(_cuda(A), _cuda(B))
    A1 = numpy.concatenate([A.astype(float), numpy.ones((rows, 1))], 1)
    B1 = B.astype(float)
    assert got.shape == (K + 1, N)
    n = min(rows, 256) + (rows + 255) // 256
    assert (abs(got - A1.T @ B1) <= n * U * (abs(A1).T @ abs(B1))).all()
