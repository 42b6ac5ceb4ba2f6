"""Launch options that a kernel does not have are refused, not dropped."""
import ctypes

import numpy as np
import pytest

from activemodelbplus.integrator import _native as N


@pytest.mark.parametrize("entry,kernel", [("amb_step_f64_ex", 0), ("amb_step_f64_ex", 1), ("amb_step_f32_ex", 0),
                                          ("amb_step_f32_ex", 2)])
def test_abi_refuses_wide_tiles_elsewhere(entry, kernel):
    """AMB_FLAG_TILE_COLS_64 away from the FP32 tile kernel (no step is asked for, so nothing is launched)."""
    lib = N.lib()
    s, m = N.amb_stencil(1e-3, 1, 1), N.amb_model(0, 0, 0, 0, 0, 0, 0)
    cfg = N.amb_kernel_config(kernel, 16, 1, N.AMB_FLAG_TILE_COLS_64)
    residual = (None,) if entry == "amb_step_f32_ex" else ()
    rc = getattr(lib, entry)(ctypes.byref(s), ctypes.byref(m), 0, 128, 128, 1 << 20, 2 << 20, *residual, 0, 0, None,
                             ctypes.byref(cfg), None, None)
    assert rc == N.AMB_ERR_INVALID and "AMB_FLAG_TILE_COLS_64" in N.last_error()


@pytest.mark.gpu
@pytest.mark.parametrize("precision,kernel,cols", [("f32", "tile", 48), ("f32c", "tile", 0), ("f64", "tile", 64),
                                                   ("f32", "sliding", 64)])
def test_python_refuses_other_widths(precision, kernel, cols):
    from activemodelbplus.integrator import Integrator, Model, Stencil
    with pytest.raises(ValueError, match="tile_cols"):
        Integrator(np.zeros((16, 128)), Stencil(1e-3, 1, 1), Model(), precision=precision, kernel=kernel,
                   launch={"tile_cols": cols})


@pytest.mark.gpu
def test_what_ran_still_runs():
    """Heights above 64 rows and FP64 tiles with a height were always taken."""
    from activemodelbplus.integrator import Integrator, Model, Stencil
    f = np.random.default_rng(0).normal(-0.4, 0.1, (130, 128))
    for precision in ("f32", "f64"):
        fields = []
        for launch in ({}, {"seg_rows": 100}, {"tile_cols": 32}):
            sim = Integrator(f, Stencil(1e-3, 1, 1), Model(T=0.05), precision=precision, seed=1, kernel="tile", launch=launch)
            sim.run(2)
            fields.append(sim.field)
        assert np.array_equal(fields[0], fields[1]) and np.array_equal(fields[0], fields[2])
