"""The FP64 step's workspace stays a small part of the device, whatever the grid's shape."""
import ctypes

import numpy as np
import pytest

from activemodelbplus.integrator import _native as N


def test_at_most_two_gib():
    lib = N.lib()
    for ny in (1, 16, 47, 48, 64, 100, 1000, 1 << 20, 1 << 30):
        for nx in (1, 1000, 87381, 87382, 100000, 699050, 699051, 1 << 20, 10 ** 7, 1 << 26, 1 << 30):
            if ny * nx > 1 << 36:
                continue
            need = lib.amb_step_workspace_bytes(N.AMB_F64, ny, nx)
            assert need <= 2 << 30
            if nx <= 87381:
                assert 0 < need <= (256 << 20) + 256
            if nx <= 600000:
                assert need > 0


def test_no_workspace_needs_none():
    """A shape without one: NULL is taken (no step is asked for, so nothing is launched)."""
    lib = N.lib()
    s, m, where = N.amb_stencil(1e-3, 1, 1), N.amb_model(0, 0, 0, 0, 0, 0, 0), ctypes.c_int(5)
    assert lib.amb_step_workspace_bytes(N.AMB_F64, 64, 1 << 26) == 0
    assert lib.amb_step_f64_ws(ctypes.byref(s), ctypes.byref(m), 0, 64, 1 << 26, 1 << 20, 2 << 20, 0, 0, None, None, 0, None,
                               ctypes.byref(where)) == 0
    assert where.value == 0


@pytest.mark.gpu
@pytest.mark.parametrize("nx", [100000, 750000])
def test_long_rows(nx):
    """In bands of 48 rows (a workspace of 410 MB) and without one: the tile kernel's bits."""
    from activemodelbplus.integrator import Integrator, Model, Stencil
    st, m = Stencil(1e-3, 1, 1), Model(-0.25, 0, 0.25, 1, -1, -4, 0.05)
    f = np.random.default_rng(1).normal(-0.4, 0.1, (60, nx))
    a, b = Integrator(f, st, m, seed=1), Integrator(f, st, m, seed=1, kernel="tile")
    a.run(2)
    b.run(2)
    assert np.array_equal(a.field, b.field)
