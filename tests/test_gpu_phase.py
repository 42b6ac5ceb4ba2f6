"""The FP64 step kernels behind amb_step_f64_ws (one tile per SM on small grids, three grid-wide phases
on the others) against the oracle and the tile kernel."""
import ctypes

import numpy as np
import pytest

import oracle
from activemodelbplus.integrator import Integrator, Model, Stencil
from activemodelbplus.integrator import _native as N

# tiles: one site, grids narrower than the stencils and than a tile, partial tiles, tall and wide grids;
# phases: blocks of 32 columns with and without remainder, more rows than warps and fewer
SHAPES = [(1, 1), (2, 7), (9, 31), (33, 64), (65, 33), (20, 257), (300, 40), (6000, 9), (3, 15000),
          (250, 260), (11, 7001), (20000, 7)]


def _params(T):
    m = Model(a=-0.25, b=0.1, c=0.25, kappa=1, lamb=-1, zeta=-4, T=T)
    p = oracle.Params(dt=1e-3, dx=1.0, dy=1.25, a=-0.25, b=0.1, c=0.25, kappa=1, lamb=-1, zeta=-4, T=T)
    return Stencil(dt=1e-3, dx=1.0, dy=1.25), m, p


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
def test_matches_oracle(shape):
    st, m, p = _params(0.0)
    f = np.random.default_rng(1).normal(-0.4, 0.1, shape)
    sim = Integrator(f, st, m)
    assert sim._workspace is not None
    sim.run(5)
    ref = oracle.run(f, p, 5)
    assert np.abs(sim.field - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
def test_injected_noise_matches_oracle(shape):
    import torch
    st, m, p = _params(0.05)
    rng = np.random.default_rng(2)
    f, xi = rng.normal(-0.4, 0.1, shape), rng.standard_normal((3, 2) + shape)
    ny, nx = shape
    a = torch.from_numpy(f.copy()).cuda()
    b, x = torch.empty_like(a), torch.from_numpy(xi).cuda()
    nbytes = N.lib().amb_step_workspace_bytes(N.AMB_F64, ny, nx)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    s, mm, where = N.stencil_struct(st), N.model_struct(m), ctypes.c_int()
    rc = N.lib().amb_step_f64_ws(ctypes.byref(s), ctypes.byref(mm), 0, ny, nx, a.data_ptr(), b.data_ptr(), 0, 3,
                                 x.data_ptr(), ws.data_ptr(), nbytes, torch.cuda.current_stream().cuda_stream,
                                 ctypes.byref(where))
    assert rc == 0 and where.value == 1
    ref = oracle.run(f, p, 3, noise="injected", injected=xi)
    assert np.abs(b.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.gpu
@pytest.mark.parametrize("shape,T", [(s, 0.05) for s in SHAPES] + [((2050, 2100), 0.05), ((2050, 2100), 0.0)])
def test_same_bits_as_the_tile_kernel(shape, T):
    """Philox noise; the last grid exceeds the workspace, so it is walked in bands of rows."""
    st, m, _ = _params(T)
    f = np.random.default_rng(3).normal(-0.4, 0.1, shape)
    a, b = Integrator(f, st, m, seed=9), Integrator(f, st, m, seed=9, kernel="tile")
    for n in (2, 1):
        a.run(n)
        b.run(n)
    assert np.array_equal(a.field, b.field)


def test_workspace_arguments_are_checked():
    lib = N.lib()
    s, m = N.amb_stencil(1e-3, 1, 1), N.amb_model(0, 0, 0, 0, 0, 0, 0)
    need = lib.amb_step_workspace_bytes(N.AMB_F64, 64, 64)
    assert need >= 64 * 64 * 8 * 8
    assert lib.amb_step_workspace_bytes(N.AMB_F64, 8192, 8192) <= (256 << 20) + 256
    for ws, size in ((None, need), (4096, need - 1), (4100, need)):
        assert lib.amb_step_f64_ws(ctypes.byref(s), ctypes.byref(m), 0, 64, 64, 1 << 20, 2 << 20, 0, 1, None, ws, size,
                                   None, None) == N.AMB_ERR_INVALID
