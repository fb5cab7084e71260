"""BoundaryNet.gradient takes its targets as torch takes them: broadcast to the outputs' shape, in any
floating type, as a function in reverse and in forward mode; shapes that do not fit are refused."""
import numpy
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _net(B=33):
    from opencl_fdtd_gb300 import learned_boundary as lb
    gen = torch.Generator(device="cuda").manual_seed(B)
    net = lb.BoundaryNet(seed=1)
    return net, *(torch.randn((B, n), generator=gen, device="cuda") for n in (lb.IN, lb.OUT))


@pytest.mark.parametrize("shape", [(33, 7), (33, 3), (32, 6), (2, 32, 6)])
def test_targets_of_another_shape_are_refused(shape):
    net, X, _ = _net()
    with pytest.raises(RuntimeError):
        net.gradient(0, X, torch.zeros(shape, device="cuda"))


@pytest.mark.parametrize("weighted", [True, False])
def test_forward_mode_of_the_loss(weighted):
    from torch.autograd import forward_ad
    net, X, T = _net()
    V = torch.randn_like(T)
    Tr = T.clone().requires_grad_(True)
    loss, grad = net.gradient(2, X, Tr, weighted)
    loss.backward()
    grad = grad.clone()
    with forward_ad.dual_level():
        out, g = net.gradient(2, X, forward_ad.make_dual(T, V), weighted)
        value, tangent = forward_ad.unpack_dual(out)
        assert tangent is not None
        assert torch.equal(g, grad) and torch.equal(value, loss.detach())
        # two float32 sums of the same 198 products
        terms = (Tr.grad * V).abs().sum()
        assert (tangent - (Tr.grad * V).sum()).abs() <= 2 * (T.numel() + 8) * 2.0 ** -24 * terms


@pytest.mark.parametrize("dtype", [torch.float64, torch.float16])
def test_targets_of_another_type(dtype):
    net, X, T = _net()
    T = T.to(dtype)
    loss, grad = net.gradient(1, X, T.to(torch.float32))
    loss, grad = loss.clone(), grad.clone()
    other, g = net.gradient(1, X, T)
    assert torch.equal(g, grad)
    # the loss as torch forms it, in the type torch gives it: two sums of the same 198 squares
    assert other.dtype == torch.promote_types(torch.float32, dtype)
    assert abs(float(other) - float(loss)) <= 2 * (T.numel() + 8) * 2.0 ** -24 * float(loss)


@pytest.mark.parametrize("shape", [(6,), (1, 6), (33, 1)])
def test_targets_are_broadcast(shape):
    net, X, _ = _net()
    T = torch.linspace(-1, 1, int(numpy.prod(shape)), device="cuda").reshape(shape)
    loss, grad = net.gradient(4, X, T)
    loss, grad = loss.clone(), grad.clone()
    full, g = net.gradient(4, X, T.expand(33, 6).contiguous())
    assert torch.equal(g, grad) and torch.equal(full, loss)


def test_targets_with_a_further_dimension():
    net, X, T = _net()
    zero = net.gradient(5, X, torch.zeros_like(T))[1].clone()
    loss, grad = net.gradient(5, X, torch.stack([T, -T]))
    grad = grad.clone()
    assert torch.equal(grad, zero)                           # the mean of the two targets is exactly zero
    both = [float(net.gradient(5, X, t)[0]) for t in (T, -T)]
    assert abs(float(loss) - sum(both) / 2) <= 4 * (2 * T.numel() + 8) * 2.0 ** -24 * float(loss)
