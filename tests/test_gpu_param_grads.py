"""Parameter gradients in the weights' layout (amb_conv5x5_param_grads) and the operand images
(amb_conv5x5_images)."""
import numpy as np
import pytest

import oracle.learned as OL

pytestmark = pytest.mark.gpu

LAYERS = [(32, 32, 32, 32), (5, 16, 32, 32), (32, 32, 2, 16), (7, 16, 9, 16)]


# a single row block and remainders of 4 and 8 rows, one and several windows, more row blocks than CTAs
@pytest.mark.parametrize("shape", [(1, 3, 128), (2, 13, 128), (1, 20, 256), (3, 130, 384)])
@pytest.mark.parametrize("cin_used,cin,cout,npad", LAYERS)
def test_param_grads(shape, cin_used, cin, cout, npad):
    """Against the FP64 oracle to FP32 accumulation (2e-5 of the largest gradient, as amb_conv5x5_wgrad)."""
    import torch
    from activemodelbplus import learned as L
    B, H, W = shape
    rng = np.random.default_rng(H + cin + npad)
    x = OL.bf16_round(rng.standard_normal((B, cin_used, H, W)))
    dz = OL.bf16_round(rng.standard_normal((B, cout, H, W)))
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    gw, gb = L.param_grads(L.to_chunks(torch.from_numpy(x).float().cuda(), cin),
                           L.to_chunks(torch.from_numpy(dz).float().cuda(), npad), cin=cin, npad=npad,
                           cin_used=cin_used, cout=cout, scratch=L._Scratch(), error=err)
    assert int(err.item()) == 0
    _, ref = OL.conv5x5_grads(x, np.zeros((cout, cin_used, 5, 5)), dz)
    assert np.abs(gw.cpu().numpy() - ref).max() < 2e-5 * max(1.0, np.abs(ref).max())
    rb = dz.sum(axis=(0, 2, 3))
    assert np.abs(gb.cpu().numpy()[:cout] - rb).max() < 2e-5 * max(1.0, np.abs(rb).max())
    assert not gb[cout:].any()


@pytest.mark.parametrize("cin_used,cin,cout,npad", LAYERS)
def test_images(cin_used, cin, cout, npad):
    import torch
    from activemodelbplus import learned as L
    from activemodelbplus.integrator import _native as N
    w = torch.randn(cout, cin_used, 5, 5, device="cuda")
    img, dimg = (torch.empty(25 * cin * npad, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    assert N.lib().amb_conv5x5_images(w.data_ptr(), cout, cin_used, cin, npad, img.data_ptr(), dimg.data_ptr(),
                                      torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(img, L.weight_image(w, cin, npad).reshape(-1))
    assert torch.equal(dimg, L.dgrad_image(w, cin, npad).reshape(-1))


@pytest.mark.parametrize("layers", [2, 3, 9])
@pytest.mark.parametrize("shape", [(1, 3, 128), (3, 13, 256)])
def test_stack_equals_the_layers(shape, layers):
    """One call for all layers: bitwise the layers' own calls (images of more layers than one launch takes,
    activations that take turns, gradients handed down through two buffers)."""
    import torch
    from activemodelbplus import learned as L
    from activemodelbplus.integrator import _native as N
    B, H, W = shape
    g = torch.Generator(device="cuda").manual_seed(layers)
    net = L.FluxNet(seed=5, layers=layers)
    for b in net.biases[:-1]:
        b.normal_(0, 0.1, generator=g)
    x = torch.randn(B, 2, H, W, 8, device="cuda", generator=g).to(torch.bfloat16)
    dflux = torch.randn(B, 2, H, W, device="cuda", generator=g)
    flux = net.forward(x, train=True)
    gw, gb = net.backward(dflux)
    assert torch.equal(net.forward(x), flux)
    img = [L.weight_image(w, net.cin[l], net.npad[l]) for l, w in enumerate(net.weights)]
    dimg = [None] + [L.dgrad_image(net.weights[l], net.cin[l], net.npad[l]) for l in range(1, layers)]
    acts, pres = [x], []
    for l in range(layers - 1):
        out = torch.empty(B, 4, H, W, 8, dtype=torch.bfloat16, device="cuda")
        pres.append(torch.empty_like(out))
        L.conv_forward(acts[-1], img[l], net.biases[l], cin=net.cin[l], npad=32, epilogue=N.AMB_EPI_GELU, out=out, pre=pres[-1])
        acts.append(out)
    want = torch.empty_like(flux)
    L.conv_forward(acts[-1], img[-1], net.biases[-1], cin=32, npad=16, cout=2, epilogue=N.AMB_EPI_F32, out_f32=want)
    assert torch.equal(flux, want)
    dz = L.to_chunks(dflux, 16)
    for l in range(layers - 1, -1, -1):
        rw, rb = L.param_grads(acts[l], dz, cin=net.cin[l], npad=net.npad[l], cin_used=net.cin_used[l], cout=net.cout[l],
                               scratch=L._Scratch())
        assert torch.equal(gw[l], rw)
        if l == layers - 1:
            assert torch.allclose(gb[l][:2], dflux.sum(dim=(0, 2, 3)), rtol=1e-5, atol=1e-3) and not gb[l][2:].any()
        else:
            assert torch.equal(gb[l], rb)
        if l:
            prev = torch.empty(B, 4, H, W, 8, dtype=torch.bfloat16, device="cuda")
            L.conv_forward(dz, dimg[l], None, cin=net.npad[l], npad=32, epilogue=N.AMB_EPI_GELU_BWD, out=prev, gate=pres[l - 1])
            dz = prev
    net.check_error()
