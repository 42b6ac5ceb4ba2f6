"""The fixed-point update on four columns per thread against one column per thread (taken when a buffer is
not 16-byte aligned): the same integers, fields, inputs and flags, with wrap-around on one row and one quad,
values past the bound and fluxes that are infinite, not a number or beyond the face's limit."""
import pytest
import torch

from activemodelbplus.integrator import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("with_extra", [False, True])
@pytest.mark.parametrize("ny,nx", [(1, 4), (1, 128), (3, 132), (70, 1000), (130, 516)])
def test_quads_equal_columns(ny, nx, with_extra):
    g = torch.Generator(device="cuda").manual_seed(ny + nx)
    flux, extra = (torch.randn(2, ny, nx, device="cuda", generator=g) for _ in range(2))
    special = torch.tensor([float("nan"), float("inf"), -float("inf"), 1e30, -1e30], device="cuda")
    for t in (flux, extra):
        at = torch.randint(0, t.numel(), (5,), device="cuda", generator=g)
        t.view(-1)[at] = special
    q0 = torch.randint(-(1 << 26), 1 << 26, (ny, nx), dtype=torch.int32, device="cuda", generator=g)  # |phi| up to 4
    params = torch.tensor([-3.0, 0.5, 0.05], device="cuda")
    lib, strm, out = N.lib(), torch.cuda.current_stream().cuda_stream, []
    for off in (0, 1):  # a float of offset: columns
        q, f = q0.clone(), torch.empty(ny * nx + 1, device="cuda")[off:off + ny * nx]
        flag, step = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int64, device="cuda")
        x = torch.zeros(1, 2, ny, nx, 8, dtype=torch.bfloat16, device="cuda")
        rc = lib.amb_learned_update_input(flux.data_ptr(), extra.data_ptr() if with_extra else None, ny, nx, 0.05, 1.0, 1.25,
                                          None, 0.0, q.data_ptr(), f.data_ptr(), 3.0, flag.data_ptr(), step.data_ptr(),
                                          params.data_ptr(), x.data_ptr(), strm)
        assert rc == 0, N.last_error()
        out.append((q, f.clone(), flag, step, x))
    assert all(torch.equal(a, b) for a, b in zip(*out))
    assert int(out[0][2]) == 1 and int(out[0][3]) == 1
