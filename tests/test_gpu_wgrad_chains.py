"""Weight and bias gradients where a CTA sums many row blocks: what one accumulator of the tensor core takes
is bounded, however large the batch."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,npad", [(32, 32), (16, 32), (32, 16), (16, 16)])
def test_error_does_not_grow_with_the_batch(cin, npad):
    """Against FP64 sums, values of one sign, some hundred row blocks per CTA: 2e-5 of the largest gradient, what
    64 truncated FP32 additions per accumulator (64 * 2^-23) and a few hundred rounded ones between them can
    leave (128 instead of 64, half the bound's first part again)."""
    import torch
    from activemodelbplus import learned as L
    B, H, W = 16, 512, 512
    g = torch.Generator(device="cuda").manual_seed(cin + npad)
    x = (0.5 + torch.randn(B, cin // 8, H, W, 8, device="cuda", generator=g)).to(torch.bfloat16)
    dz = (0.5 + torch.randn(B, npad // 8, H, W, 8, device="cuda", generator=g)).to(torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    gw, gb = L.param_grads(x, dz, cin=cin, npad=npad, cin_used=cin, cout=npad, scratch=L._Scratch(), error=err)
    assert int(err.item()) == 0
    rows = [t.double().permute(0, 1, 4, 2, 3).reshape(B, -1, H, W) for t in (x, dz)]
    zs = rows[1].reshape(B, npad, H * W)
    for ky, kx in ((0, 0), (1, 2), (4, 4)):
        xs = torch.roll(rows[0], (2 - ky, 2 - kx), (2, 3)).reshape(B, cin, H * W)
        want = torch.einsum("bin,bon->oi", xs, zs)
        assert (gw[:, :, ky, kx].double() - want).abs().max() <= 2e-5 * want.abs().max()
    want = zs.sum(dim=(0, 2))
    assert (gb.double() - want).abs().max() <= 2e-5 * want.abs().max()


# row counts with and without a remainder of 4 and of 8, fewer rows than a block, several blocks per CTA
@pytest.mark.parametrize("shape", [(1, 3, 128), (1, 12, 128), (2, 13, 128), (2, 14, 256), (3, 130, 384)])
@pytest.mark.parametrize("cin,npad", [(32, 32), (16, 32), (32, 16), (16, 16)])
def test_an_infinite_gradient_stays_infinite(shape, cin, npad):
    """One infinite gradient beside positive inputs: its channel's weight gradients are all +inf (each tap and
    input channel has that one infinite term), no other channel changes."""
    import torch
    from activemodelbplus import learned as L
    B, H, W = shape
    g = torch.Generator(device="cuda").manual_seed(H)
    x = (0.5 + torch.rand(B, cin // 8, H, W, 8, device="cuda", generator=g)).to(torch.bfloat16)
    dz = torch.randn(B, npad // 8, H, W, 8, device="cuda", generator=g).to(torch.bfloat16)
    clean = L.conv_wgrad(x, dz, cin=cin, npad=npad)
    other = [c for c in range(npad) if c != 11]
    for b, row, col in ((0, 0, 40), (B - 1, 1, 0), (0, H // 2, W - 1), (B - 1, H - 1, 127), (0, H - 2, 5)):
        z = dz.clone()
        z[b, 1, row, col, 3] = float("inf")  # channel 11
        dw = L.conv_wgrad(x, z, cin=cin, npad=npad)
        assert bool((dw[:, :, 11] == float("inf")).all())
        assert torch.equal(dw[:, :, other], clean[:, :, other])


def test_gradients_at_any_float():
    """The caller's gradient arrays need no more than a float's alignment."""
    import torch
    from activemodelbplus import learned as L
    from activemodelbplus.integrator import _native as N
    lib, stream = N.lib(), torch.cuda.current_stream().cuda_stream
    x, dz = (torch.randn(1, 4, 8, 128, 8, device="cuda").to(torch.bfloat16) for _ in range(2))
    nbytes = lib.amb_conv5x5_wgrad_scratch_bytes(1, 8, 128, 32, 32)
    scratch = torch.empty(nbytes // 4, device="cuda")
    dw, gw, gb = torch.zeros(25 * 1024 + 3, device="cuda"), torch.zeros(25 * 1024 + 1, device="cuda"), torch.zeros(33, device="cuda")
    for at in (1, 2, 3):
        assert lib.amb_conv5x5_wgrad(x.data_ptr(), dz.data_ptr(), 1, 8, 128, 32, 32, dw[at:].data_ptr(), scratch.data_ptr(),
                                     nbytes, None, stream) == 0, N.last_error()
        assert torch.equal(dw[at:at + 25 * 1024].reshape(25, 32, 32), L.conv_wgrad(x, dz, cin=32, npad=32))
    assert lib.amb_conv5x5_param_grads(x.data_ptr(), dz.data_ptr(), 1, 8, 128, 32, 32, 32, 32, gw[1:].data_ptr(),
                                       gb[1:].data_ptr(), scratch.data_ptr(), nbytes, None, stream) == 0, N.last_error()
    assert torch.equal(gw[1:].reshape(32, 32, 5, 5), L.wgrad_to_weights(L.conv_wgrad(x, dz, cin=32, npad=32), 32, 32))
