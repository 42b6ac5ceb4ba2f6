"""Operand images follow the shapes that the weights have, not those that the network was made with."""
import pytest

pytestmark = pytest.mark.gpu


def test_narrower_weights_are_padded_with_zeros():
    """Layers with fewer channels give what the same weights give in zeros of the full shape."""
    import torch
    from activemodelbplus import learned as L
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(2, 2, 16, 128, 8, device="cuda", generator=g).to(torch.bfloat16)
    dflux = torch.randn(2, 2, 16, 128, device="cuda", generator=g)
    nets = [L.FluxNet(seed=3, layers=3) for _ in range(2)]
    for l, (cout, cin) in enumerate([(20, 3), (32, 20), (1, 30)]):
        w = nets[0].weights[l]
        narrow = w[:cout, :cin].clone()
        nets[1].weights[l] = narrow
        w.zero_()
        w[:cout, :cin] = narrow
    out = []
    for net in nets:
        net.refresh()
        flux = net.forward(x, train=True)
        out.append([flux] + net.backward(dflux)[0])
        net.check_error()
    for a, b in zip(*out):
        assert torch.equal(a, b)


@pytest.mark.parametrize("shape", [(33, 5, 5, 5), (32, 17, 5, 5), (32, 5, 3, 3), (32, 5, 25)])
def test_other_shapes_are_refused(shape):
    import torch
    from activemodelbplus import learned as L
    from activemodelbplus.integrator import CudaException
    net = L.FluxNet(seed=3, layers=2)
    x = torch.randn(1, 2, 16, 128, 8, device="cuda").to(torch.bfloat16)
    flux = net.forward(x)
    net.weights[0] = torch.zeros(shape, device="cuda")
    with pytest.raises((ValueError, RuntimeError, CudaException)):
        net.refresh()
    assert torch.equal(net.forward(x), flux)  # the images are those of before
